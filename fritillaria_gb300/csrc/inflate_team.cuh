// The team form of the member inflate: a CTA works on one member at a time,
// every lane decoding.  Included by inflate.cu, whose serial form it falls
// back to.
//
// What bounds the one-chain form is that 1 of 32 lanes does the Huffman
// decode: ~57 warp instructions a symbol, ~140 cycles a symbol for a member
// alone.  A DEFLATE block can be decoded from any bit: a decoder started at a
// wrong place falls into step with the true symbol boundaries after a few
// dozen codes (on short-read, FASTQ, FASTA and BCF members 1-4% of starts are
// still out of step after 512 bits, 0.03-0.2% after 1,024; codes of one length
// may never fall into step, see settle).  So the team cuts a block into one
// segment per lane and goes over it three times:
//
//   1. sync:  a lane starts SYNC_BITS before its segment and runs to the
//             segment's first symbol boundary, its presumed start;
//   2. count: a lane runs its segment from that start, counting output
//             bytes, to the next segment's first boundary.  Where that
//             is not the next lane's presumed start, the next lane counts
//             again from it, until the chain from the block's first symbol to
//             the end-of-block code is proven;
//   3. emit:  with the counts summed over the team, each lane runs its
//             segment again, writing literals to their places in the member's
//             output, held whole in shared memory, and leaving each match as
//             a 3-byte token (length, distance) in its own destination, its
//             first byte marked in a bitmap.
//
// One step of a pass takes one code with no branch in it: the 32-bit window at
// the lane's bit position, one table lookup, and the table entry says how many
// bits to drop, how many bytes come out and which table comes next (the
// literal/length root, a second-level table, a length's extra bits, the
// distance root).  Lanes at literals, lengths and distances so run the same
// instructions.  Stores are predicated by hand: branches that split a warp, and
// loads whose latency every step waits for, were what the first forms spent
// their time on.  The compressed words of a round are staged in shared memory
// by cp.async for the same reason (read through L1 a step took 250-400 cycles,
// staged 130).
//
// Matches are copied once the whole member is decoded (nothing in the decode
// reads the output; copy_matches).  Then the CRC-32 is taken from shared memory
// and the member is written with 16-byte stores.
//
// Anything out of the ordinary (an invalid or truncated stream, a member over
// 64 KiB, a code whose tables do not fit) goes to the serial form from the
// member's start, whose checks and statuses are the reference's; so do, in a
// launch of many, members of short blocks (BRIEF).
//
// Measured on GB300 against the serial form (its tuned shape, the inflate alone):
// 1M short reads 8.7 -> 2.48 ms (119 GB/s of output), ultra-long reads 6.3 ->
// 1.26 ms, BCF 3.6 -> 0.78 ms, FASTQ 4.6 -> 1.13 ms, FASTA 3.3 -> 0.63 ms; one
// short-read member alone 4.4 -> 0.139 ms.  No one unit bounds it with the SMs
// full: 24 warps an SM issue 63% of the time (the ALU pipe 63% busy), and for
// each instruction a warp waits 1.9 cycles for its own last result, 1.9 at
// barriers, 1.4 for shared memory (40% of whose wavefronts are bank conflicts),
// 1.2 for another warp and 0.9 for the ALUs; 403,000 warp instructions a
// short-read member, DRAM under 3%.  Twelve warps: ten and eleven measured
// even to 3% slower, sixteen slower (the sync pass grows with the lanes), and
// 192 to 320 decoding lanes of the twelve warps' 384 0-10% slower.  Two CTAs
// fill the shared memory; one alone gives two thirds of the rate.
#pragma once

namespace team {

constexpr u32 LR = 9, DR = 8;           // literal/length and distance roots
constexpr u32 LIT_CAP = 852;            // entries of the largest 9-bit-root code of 286 symbols
constexpr u32 DIST_AT = LIT_CAP;        // distance tables follow
constexpr u32 DIST_CAP = 256 + 384;     // root and second level (a code that needs more goes to the serial form)
constexpr u32 EXTRA_AT = DIST_AT + DIST_CAP;
constexpr u32 EXTRA_CAP = 248;          // four length symbols for each of 1..5 extra bits
constexpr u32 TAB = EXTRA_AT + EXTRA_CAP;
static_assert(TAB <= 2048, "an entry holds an 11-bit table index");

constexpr u32 OUT_MAX = 65536; // a BGZF member's largest output

// Table entry:
//   [1:0]   1 end of block, 2 distance, 3 no valid code; 0 anything else
//   [12:2]  index of the next code's table
//   [17:13] 32 minus that table's index bits
//   [26:18] output bytes: 1 literal, 3..258 length, 0 anything else
//   [31:27] bits to drop
constexpr u32 F_END = 1, F_DIST = 2, F_BAD = 3;
__host__ __device__ constexpr u32 entry(u32 bits, u32 bytes, u32 next, u32 width, u32 flags)
{
    return (bits << 27) | (bytes << 18) | (((32u - width) & 31u) << 13) | (next << 2) | flags;
}
__host__ __device__ constexpr u32 to_lit(u32 bits, u32 bytes, u32 flags) { return entry(bits, bytes, 0, LR, flags); }
__host__ __device__ constexpr u32 to_dist(u32 bits, u32 bytes) { return entry(bits, bytes, DIST_AT, DR, 0); }

struct Code {
    u32 cnt[16];
    u32 lim[16];  // first 15-bit code past those of each length (left-aligned)
    u32 offs[16]; // index in `sorted` of each length's first symbol
    u32 n;        // symbols with a code
};

constexpr u32 STAGE_WORDS = 6272; // compressed words of one round: 25 KiB, past the largest default zlib block of the shapes above
// A lane runs at most one symbol (48 bits) past its segment and loads up to
// three words ahead.
constexpr u32 ROUND_BITS = 32u * (STAGE_WORDS - 6);
constexpr u32 HEAD_BITS = 2304;   // code lengths of a dynamic block: at most 316 symbols of at most 7 bits each
constexpr u32 MARKS = (OUT_MAX + 16 + 255) / 256 * 8; // words of one mark per output byte, whole groups
constexpr u32 GROUP_MATCHES = 256 / 3 + 1; // most matches that start in 256 bytes

// Places in `out` and `starts` count from the first byte of `out`; the
// member's first byte lies at its HBM address modulo 16.
template <int NW> struct Smem {
    static constexpr u32 NT = 32 * NW;
    static constexpr u32 WIN = 256 * NW; // bytes of a copy window: a group a warp (two measured 2% slower)
    alignas(16) u8 out[OUT_MAX + 16]; // the member's output, at the alignment of its place in HBM
    u32 starts[MARKS];                // first bytes of matches
    u32 tab[TAB];
    u32 val[EXTRA_AT]; // beside tab: a literal's byte; a distance's base - 1 | (32 - extra bits) << 26
    union {
        u32 stage[STAGE_WORDS]; // decoding: the round's compressed words
        u16 back[2 * WIN];      // copying: a byte's distance back to the one it copies
        u32 crc[4][256]; // checking
    };
    u32 end[NT]; // copying: each warp's list of a group's matches
    u32 wa[NW], wb[NW];
    Code lit, dist;
    u32 sh[8]; // uniform values handed from one thread to the team
    u32 fail, hint;
    u32 brief, blocks; // bits a block below which the member is the serial form's; its blocks so far
    u32 list[NW], listed; // members that wait for the serial form
    u32 q, q_end, streak; // the CTA's place in the queue, and members in a row that the team did not take
    u16 lsorted[288], dsorted[32];
    u8 lens[320];
};

// ---- shared memory by 32-bit address ------------------------------------------
__device__ __forceinline__ u32 lds32(u32 a)
{
    u32 v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ u32 lds8(u32 a)
{
    u32 v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ u32 lds16_if(u32 p, u32 a) // 0 where not
{
    u16 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tmov.u16 %0, 0;\n\t@p ld.shared.u16 %0, [%2];\n\t}" : "=h"(v) : "r"(p), "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts16(u32 a, u32 v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((u16)v) : "memory"); }
__device__ __forceinline__ void sts32(u32 a, u32 v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts32_if(u32 p, u32 a, u32 v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.u32 [%1], %2;\n\t}" ::"r"(p), "r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts16_if(bool p, u32 a, u32 v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.u16 [%1], %2;\n\t}" ::"r"((u32)p), "r"(a), "h"((u16)v) : "memory");
}
__device__ __forceinline__ void sts8(u32 a, u32 v) { asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts8_if(bool p, u32 a, u32 v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.u8 [%1], %2;\n\t}" ::"r"((u32)p), "r"(a), "r"(v) : "memory");
}
// v to the first n (0, or any number) of eight halves.
__device__ __forceinline__ void sts16_run(u32 a, u32 n, u32 v)
{
    asm volatile("{\n\t.reg .pred p<8>;\n\t"
                 "setp.gt.u32 p0, %1, 0;\n\tsetp.gt.u32 p1, %1, 1;\n\tsetp.gt.u32 p2, %1, 2;\n\tsetp.gt.u32 p3, %1, 3;\n\t"
                 "setp.gt.u32 p4, %1, 4;\n\tsetp.gt.u32 p5, %1, 5;\n\tsetp.gt.u32 p6, %1, 6;\n\tsetp.gt.u32 p7, %1, 7;\n\t"
                 "@p0 st.shared.u16 [%0], %2;\n\t@p1 st.shared.u16 [%0+2], %2;\n\t@p2 st.shared.u16 [%0+4], %2;\n\t"
                 "@p3 st.shared.u16 [%0+6], %2;\n\t@p4 st.shared.u16 [%0+8], %2;\n\t@p5 st.shared.u16 [%0+10], %2;\n\t"
                 "@p6 st.shared.u16 [%0+12], %2;\n\t@p7 st.shared.u16 [%0+14], %2;\n\t}" ::"r"(a), "r"(n), "h"((u16)v)
                 : "memory");
}
__device__ __forceinline__ u32 lds8_if(bool p, u32 a) // 0 where not
{
    u32 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tmov.u32 %0, 0;\n\t@p ld.shared.u8 %0, [%2];\n\t}" : "=r"(v) : "r"((u32)p), "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ u32 lds32_if(bool p, u32 a) // 0 where not
{
    u32 v;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tmov.u32 %0, 0;\n\t@p ld.shared.u32 %0, [%2];\n\t}" : "=r"(v) : "r"((u32)p), "r"(a) : "memory");
    return v;
}
// A match's token in its first three bytes, and its mark.
__device__ __forceinline__ void token_if(bool p, u32 a, u32 token, u32 mark_at, u32 mark)
{
    asm volatile("{\n\t.reg .pred p;\n\t.reg .u32 t;\n\tsetp.ne.u32 p, %0, 0;\n\t"
                 "@p st.shared.u8 [%1], %2;\n\tshr.u32 t, %2, 8;\n\t@p st.shared.u8 [%1+1], t;\n\t"
                 "shr.u32 t, %2, 16;\n\t@p st.shared.u8 [%1+2], t;\n\t@p red.shared.or.b32 [%3], %4;\n\t}" ::"r"((u32)p),
                 "r"(a), "r"(token), "r"(mark_at), "r"(mark)
                 : "memory");
}
// ---- end

__device__ __forceinline__ u32 shr_clamp(u32 v, u32 n)
{
    u32 r;
    asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));
    return r;
}

// A lane's place in the staged words and the tables.  `a` counts bits from the
// first staged word; the word after the next is loaded one refill ahead.
struct Walk {
    u32 a, lo, hi, nx, wa, b4, t;
    __device__ __forceinline__ void start(u32 stage, u32 at)
    {
        a = at;
        wa = stage + 4u * (a >> 5);
        lo = lds32(wa);
        hi = lds32(wa + 4);
        nx = lds32(wa + 8);
        wa += 12;
        b4 = 0;
        t = 32u - LR;
    }
    // Past a word boundary (`moved` > 31): the next word, predicated.
    __device__ __forceinline__ void refill(u32 moved)
    {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.u32 p, %4, 31;\n\t@p mov.u32 %0, %1;\n\t@p mov.u32 %1, %2;\n\t"
                     "@p ld.shared.u32 %2, [%3];\n\t@p add.u32 %3, %3, 4;\n\t}"
                     : "+r"(lo), "+r"(hi), "+r"(nx), "+r"(wa)
                     : "r"(moved)
                     : "memory");
    }
    // One code: its entry, and past it.
    __device__ __forceinline__ u32 step(u32 tab)
    {
        const u32 e = lds32(place(tab, window()));
        pass(e);
        return e;
    }
    // The same, with `w` the 32 bits from the code on and `v` the value beside its entry.
    __device__ __forceinline__ u32 step(u32 tab, u32 value, u32 &w, u32 &v)
    {
        w = window();
        const u32 at = place(tab, w), e = lds32(at);
        v = lds32(at + value);
        return e;
    }
    __device__ __forceinline__ u32 window() const { return __funnelshift_r(lo, hi, a); }
    __device__ __forceinline__ u32 place(u32 tab, u32 w) const
    {
        return tab + b4 + 4u * __funnelshift_r(__funnelshift_l(0u, w, t), 0u, t);
    }
    __device__ __forceinline__ void pass(u32 e)
    {
        const u32 na = a + (e >> 27);
        refill(na ^ a);
        a = na;
        b4 = e & 0x1ffcu;
        t = e >> 13;
    }
};

// What a code puts into the output: a literal's byte at `o`, or at a distance
// the token of its match, whose length came before.
__device__ __forceinline__ void emit_code(u32 out, u32 starts, u32 e, u32 v, u32 w, u32 &o, u32 &ml)
{
    const u32 n = (e >> 18) & 511u;
    sts8_if(n == 1u, out + o, v);
    if (n) ml = n;
    o += n;
    const u32 md = o - ml; // at a distance: the match's first byte
    const u32 token = (v & 0x7fffu) + shr_clamp(w << (32u - (e >> 27)), v >> 26) + ((ml - 3u) << 15);
    token_if((e & 2u) != 0u, out + md, token, starts + ((md >> 5) << 2), 1u << (md & 31u));
}

__device__ __forceinline__ u32 length_entry(u32 sym, u32 L)
{
    const u32 i = sym - 257;
    if (i < 8) return to_dist(L, 3 + i);
    if (i == 28) return to_dist(L, 258);
    const u32 x = (i - 4) >> 2;
    return entry(L, 0, EXTRA_AT + 4u * ((1u << x) - 2u) + (((i & 3u)) << x), x, 0);
}

// The entry of literal/length symbol `sym` with a code of L bits.
__device__ __forceinline__ u32 lit_entry_of(u32 sym, u32 L)
{
    if (sym < 256) return to_lit(L, 1, 0);
    if (sym == 256) return to_lit(L, 0, F_END);
    if (sym > 285) return to_lit(1, 0, F_BAD);
    return length_entry(sym, L);
}

__device__ __forceinline__ u32 dist_entry_of(u32 sym, u32 L)
{
    if (sym >= 30) return to_lit(1, 0, F_BAD);
    const u32 x = sym < 4 ? 0u : (sym - 2u) >> 1;
    return to_lit(L + x, 0, F_DIST);
}

__device__ __forceinline__ u32 dist_value_of(u32 sym)
{
    const u32 x = sym < 4 ? 0u : (sym - 2u) >> 1;
    const u32 b = sym < 4 ? sym : ((2u + (sym & 1u)) << x);
    return b | ((32u - x) << 26);
}

// The two codes' counts, limits, offsets and symbols in order, by the team:
// a warp takes a code length (or two) and finds its symbols by ballots.  False
// (uniform): over-subscribed, or incomplete in a form these tables do not take.
template <int NW> __device__ __forceinline__ bool code_order(Smem<NW> *sm, u32 nlen, u32 ndist)
{
    const u32 lane = lane_id(), warp = threadIdx.x / 32;
    constexpr u32 K = 9; // 288 / 32
    u32 L[K];
#pragma unroll
    for (u32 k = 0; k < K; ++k) L[k] = 32u * k + lane < nlen ? sm->lens[32u * k + lane] : 0u;
    const u32 D = lane < ndist ? sm->lens[nlen + lane] : 0u;
    for (u32 l = 1 + warp; l < 16; l += NW) {
        u32 c = 0;
#pragma unroll
        for (u32 k = 0; k < K; ++k) c += __popc(__ballot_sync(FRT_FULL_MASK, L[k] == l));
        const u32 d = __popc(__ballot_sync(FRT_FULL_MASK, D == l));
        if (lane == 0) {
            sm->lit.cnt[l] = c;
            sm->dist.cnt[l] = d;
        }
    }
    __syncthreads();
    // lanes 0..15 the literal/length code, 16..31 the distance code: sums over
    // the lengths, in every warp
    const u32 l = lane & 15u;
    Code *const c = lane < 16 ? &sm->lit : &sm->dist;
    const u32 mine = l ? c->cnt[l] : 0u;
    u32 lim = mine << (15 - l), off = mine;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const u32 a = __shfl_up_sync(FRT_FULL_MASK, lim, d, 16), b = __shfl_up_sync(FRT_FULL_MASK, off, d, 16);
        if ((int)l >= d) {
            lim += a;
            off += b;
        }
    }
    if (warp == 0) {
        c->lim[l] = lim;
        c->offs[l] = off - mine;
        if (l == 15) c->n = off;
    }
    const u32 first = off - mine;
    for (u32 x = 1 + warp; x < 16; x += NW) {
        u32 at = __shfl_sync(FRT_FULL_MASK, first, x);
#pragma unroll
        for (u32 k = 0; k < K; ++k) {
            const u32 m = __ballot_sync(FRT_FULL_MASK, L[k] == x);
            if (L[k] == x) sm->lsorted[at + __popc(m & lanemask_lt())] = (u16)(32u * k + lane);
            at += __popc(m);
        }
        const u32 d = __shfl_sync(FRT_FULL_MASK, first, 16 + x);
        const u32 m = __ballot_sync(FRT_FULL_MASK, D == x);
        if (D == x) sm->dsorted[d + __popc(m & lanemask_lt())] = (u16)lane;
    }
    // complete, empty, or a single code that the root resolves
    const u32 root = lane < 16 ? LR : DR;
    const u32 all = __shfl_sync(FRT_FULL_MASK, lim, lane | 15u), count = __shfl_sync(FRT_FULL_MASK, off, lane | 15u);
    const u32 in_root = __shfl_sync(FRT_FULL_MASK, off, (lane & 16u) + root);
    const bool good = all == 32768u || count == 0 || (all < 32768u && count == 1 && in_root == 1);
    const bool fine = __all_sync(FRT_FULL_MASK, good); // the same in every warp
    __syncthreads();
    return fine;
}

// The length, at most `most`, of the code that 15-bit value v opens, which is
// known to be over `from` (else past `most`).
template <u32 from, u32 most> __device__ __forceinline__ u32 code_len(const Code *c, u32 v)
{
    u32 L = from + 1; // limits grow with the length: as many as v has passed
#pragma unroll
    for (u32 l = from + 1; l <= most; ++l) L += v >= c->lim[l] ? 1u : 0u;
    return L;
}

// Second-level tables' places, by one warp: prefixes from the first that no
// code of at most `root` bits resolves, in order.  False: they do not fit.
template <u32 root> __device__ __forceinline__ bool sub_tables(u32 *tab, const Code *c, u32 at, u32 sub_at, u32 end_at)
{
    const u32 lane = lane_id();
    const u32 first = c->lim[root] >> (15 - root), size = 1u << root;
    u32 next = sub_at;
    for (u32 b = first; b < size; b += 32) {
        const u32 v = b + lane;
        u32 width = 0;
        if (v < size) {
            const u32 L = code_len<root, 15>(c, ((v + 1) << (15 - root)) - 1);
            width = L <= 15 ? L - root : 0u;
        }
        const u32 n = width ? 1u << width : 0u;
        u32 sum = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const u32 a = __shfl_up_sync(FRT_FULL_MASK, sum, d);
            if ((int)lane >= d) sum += a;
        }
        const u32 place = next + sum - n;
        next += __shfl_sync(FRT_FULL_MASK, sum, 31);
        if (next > end_at) return false;
        if (v < size)
            tab[at + (__brev(v) >> (32 - root))] = width ? entry(root, 0, place, width, 0) : to_lit(1, 0, F_BAD);
    }
    return true;
}

// Tables of the block whose code lengths lie in sm->lens, by the team.
// False (uniform): a code these tables do not take.
template <int NW> __device__ __forceinline__ bool build(Smem<NW> *sm, u32 nlen, u32 ndist)
{
    const u32 tid = threadIdx.x, warp = tid / 32;
    bool bad = false;
    if (!code_order<NW>(sm, nlen, ndist)) return false;
    if (warp == 0) bad = !sub_tables<LR>(sm->tab, &sm->lit, 0, 1u << LR, LIT_CAP);
    else if (warp == 1) bad = !sub_tables<DR>(sm->tab, &sm->dist, DIST_AT, DIST_AT + (1u << DR), DIST_AT + DIST_CAP);
    // the roots' own codes, one entry a thread (the last warps first: the
    // first two are placing the second level)
    for (u32 k = Smem<NW>::NT - 1 - tid; k < (1u << LR) + (1u << DR); k += Smem<NW>::NT) {
        const bool d = k >= (1u << LR);
        const u32 e = d ? k - (1u << LR) : k, root = d ? DR : LR;
        const Code *c = d ? &sm->dist : &sm->lit;
        const u32 v = (__brev(e) >> (32 - root)) << (15 - root);
        const u32 L = d ? code_len<0, DR>(c, v) : code_len<0, LR>(c, v);
        if (L <= root) {
            const u32 i = c->offs[L] + ((v - c->lim[L - 1]) >> (15 - L));
            if (d) {
                const u32 sym = sm->dsorted[i];
                sm->tab[DIST_AT + e] = dist_entry_of(sym, L);
                sm->val[DIST_AT + e] = dist_value_of(sym);
            } else {
                const u32 sym = sm->lsorted[i];
                u32 ent = lit_entry_of(sym, L);
                // a length whose extra bits also fit the root: they are in the
                // index, after the code, so it is resolved here
                if (sym >= 265 && sym < 285) {
                    const u32 x = (sym - 261) >> 2;
                    if (L + x <= LR)
                        ent = to_dist(L + x, ((4u + ((sym - 257) & 3u)) << x) + 3u + ((e >> L) & ((1u << x) - 1u)));
                }
                sm->tab[e] = ent;
                sm->val[e] = sym;
            }
        } else if (c->n <= 1) {
            sm->tab[d ? DIST_AT + e : e] = to_lit(1, 0, F_BAD); // no second level to write it
        }
    }
    if (__syncthreads_or(bad)) return false;
    // codes longer than the roots: each fills its entries of its prefix's table
    const u32 l0 = sm->lit.offs[LR] + (sm->lit.lim[LR] - sm->lit.lim[LR - 1] >> (15 - LR)), ln = sm->lit.n - min(sm->lit.n, l0);
    const u32 d0 = sm->dist.offs[DR] + (sm->dist.lim[DR] - sm->dist.lim[DR - 1] >> (15 - DR)), dn = sm->dist.n - min(sm->dist.n, d0);
    for (u32 k = tid; k < ln + dn; k += Smem<NW>::NT) {
        const bool d = k >= ln;
        const u32 i = d ? d0 + k - ln : l0 + k, root = d ? DR : LR;
        const Code *c = d ? &sm->dist : &sm->lit;
        u32 L = root + 1;
        while (L < 15 && i >= c->offs[L + 1]) ++L;
        const u32 v = c->lim[L - 1] + ((i - c->offs[L]) << (15 - L)); // the code, left-aligned in 15 bits
        const u32 at = (d ? DIST_AT : 0u) + (__brev(v >> (15 - root)) >> (32 - root));
        const u32 p = sm->tab[at];
        const u32 sub = (p >> 2) & 2047u, width = 32u - ((p >> 13) & 31u), m = L - root;
        const u32 low = (v >> (15 - L)) & ((1u << m) - 1u);
        const u32 sym = d ? sm->dsorted[i] : sm->lsorted[i];
        const u32 ent = d ? dist_entry_of(sym, m) : lit_entry_of(sym, m), value = d ? dist_value_of(sym) : sym;
        for (u32 j = __brev(low) >> (32 - m); j < (1u << width); j += 1u << m) {
            sm->tab[sub + j] = ent;
            sm->val[sub + j] = value;
        }
    }
    __syncthreads();
    return true;
}

// 32 staged bits from bit `a` on.
__device__ __forceinline__ u32 bits_at(const u32 *stage, u32 a)
{
    return __funnelshift_r(stage[a >> 5], stage[(a >> 5) + 1], a);
}

// The n code lengths from staged bit `a` on, into sm->lens, by the team; the
// code-length code's table is in place, and sm->sh[5] is set to the bits they
// take.  Returns 1, 0 where the serial form is to take the member, or -1 where
// they go on past SPAN bits (all uniform).
template <int NW, u32 SPAN> __device__ __forceinline__ int follow_lengths(Smem<NW> *sm, u32 a, u32 n)
{
    constexpr u32 NT = Smem<NW>::NT, PER = (SPAN + NT - 1) / NT;
    u16 *const jump = (u16 *)sm->tab;
    const u32 *const clt = sm->val;
    u16 *const place = (u16 *)(sm->val + 128);
    u8 *const value = (u8 *)(place + 512);
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid / 32;
#pragma unroll
    for (u32 k = 0; k < PER; ++k) {
        const u32 p = tid + k * NT;
        if (p < SPAN) {
            const u32 e = clt[bits_at(sm->stage, a + p) & 127u];
            jump[p] = (u16)min(p + (e & 15u) + ((e >> 4) & 15u), SPAN);
        }
    }
    if (tid == 0) {
        jump[SPAN] = (u16)SPAN;
        place[0] = 0;
    }
    __syncthreads();
    for (u32 r = 1; r < NT; r <<= 1) {
        u32 j[PER];
#pragma unroll
        for (u32 k = 0; k < PER; ++k) {
            const u32 p = tid + k * NT;
            j[k] = p < SPAN ? jump[jump[p]] : 0u;
        }
        if (tid < r && tid + r < NT) place[tid + r] = jump[place[tid]];
        __syncthreads();
#pragma unroll
        for (u32 k = 0; k < PER; ++k) {
            const u32 p = tid + k * NT;
            if (p < SPAN) jump[p] = (u16)j[k];
        }
        __syncthreads();
    }
    // thread r holds symbol r: the lengths before it, and for a repeat the
    // last symbol before it that is none
    const u32 p = place[tid];
    const u32 w = p < SPAN ? bits_at(sm->stage, a + p) : 0u, e = clt[w & 127u], sym = e >> 8;
    const u32 x = (w >> (e & 15u)) & ((1u << ((e >> 4) & 15u)) - 1u);
    const u32 rep = p >= SPAN ? 0u : (sym < 16 ? 1u : (sym == 18 ? 11u : 3u) + x);
    value[tid] = (u8)(sym < 16 ? sym : 0u);
    u32 sum = rep, from = sym != 16 ? tid + 1u : 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u32 y = __shfl_up_sync(FRT_FULL_MASK, sum, d), z = __shfl_up_sync(FRT_FULL_MASK, from, d);
        if ((int)lane >= d) {
            sum += y;
            from = max(from, z);
        }
    }
    if (lane == 31) {
        sm->wa[warp] = sum;
        sm->wb[warp] = from;
    }
    __syncthreads();
    sum += __reduce_add_sync(FRT_FULL_MASK, lane < warp ? sm->wa[lane] : 0u);
    from = max(from, __reduce_max_sync(FRT_FULL_MASK, lane < warp ? sm->wb[lane] : 0u));
    const u32 at = sum - rep;
    bool bad = false;
    if (rep && at < n) {
        bad = sum > n || from == 0;
        if (!bad) {
            const u8 v = value[from - 1];
            for (u32 i = at; i < sum; ++i) sm->lens[i] = v;
            if (sum == n) sm->sh[5] = p + (e & 15u) + ((e >> 4) & 15u);
        }
    }
    if (__syncthreads_or(bad)) return 0;
    return __syncthreads_or(tid == NT - 1 && sum < n) ? -1 : 1;
}

// The code lengths of a dynamic block, into sm->lens, by the team.  `a` is the
// staged bit after the block's three header bits and moves past the lengths.
//
// Read one symbol after another, the lengths (~280 symbols for short reads)
// are a chain of dependent lookups that took as long as the decode of the
// whole block.  Here every bit position gets the position after the symbol it
// would open, and the chain is followed by doubling: after k steps the first
// 2^k symbols' positions are known, and each position's 2^k-th successor.
// False (uniform): the serial form is to take the member.
template <int NW> __device__ __forceinline__ bool read_lengths(Smem<NW> *sm, u32 &a, u32 &nlen, u32 &ndist)
{
    constexpr u32 NT = Smem<NW>::NT;
    static_assert(NT >= 316, "a thread per symbol");
    static_assert(2 * (HEAD_BITS + 1) <= 4 * EXTRA_AT && 4 * 128 + 2 * 512 + 512 <= 4 * EXTRA_AT, "scratch in the tables' place");
    u32 *const clt = sm->val; // the tables are free until the block's are built
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid / 32;
    const u32 h = bits_at(sm->stage, a);
    nlen = (h & 31u) + 257;
    ndist = ((h >> 5) & 31u) + 1;
    const u32 ncode = ((h >> 10) & 15u) + 4, n = nlen + ndist;
    bool bad = nlen > 286 || ndist > 30;
    a += 14;
    if (warp == 0) { // the code-length code: lane i holds symbol i's length
        u32 L = 0;
        if (lane < 19) {
            // place of symbol `lane` in the order 16 17 18 0 8 7 9 6 10 5 11 4 12 3 13 2 14 1 15
            const u32 k = lane >= 16 ? lane - 16u : (lane == 0 ? 3u : (lane < 8 ? 19u - 2u * lane : 2u * lane - 12u));
            if (k < ncode) L = bits_at(sm->stage, a + 3 * k) & 7u;
        }
        u32 lim = 0, code = 0;
#pragma unroll
        for (u32 l = 1; l <= 7; ++l) {
            const u32 m = __ballot_sync(FRT_FULL_MASK, L == l);
            if (L == l) code = (lim >> (7 - l)) + __popc(m & lanemask_lt());
            lim += __popc(m) << (7 - l);
        }
        bad |= lim != 128u; // it has to be complete
        // an entry: bits of the code | extra bits << 4 | symbol << 8
        if (L && !bad)
            for (u32 j = __brev(code) >> (32 - L); j < 128u; j += 1u << L)
                clt[j] = L | ((lane == 16 ? 2u : (lane == 17 ? 3u : (lane == 18 ? 7u : 0u))) << 4) | (lane << 8);
    }
    a += 3 * ncode;
    if (__syncthreads_or(bad)) return false;
    // half the positions do for most headers (~1,000 bits for short reads)
    int got = follow_lengths<NW, HEAD_BITS / 2>(sm, a, n);
    if (got < 0) got = follow_lengths<NW, HEAD_BITS>(sm, a, n);
    if (got <= 0) return false;
    a += sm->sh[5];
    return sm->lens[256] != 0;
}

// Copies the matches of out[skew, skew + n).  Sets sm->fail (uniform) where a
// distance reaches before the member's first byte.
//
// A match may copy bytes that another one writes, chains of 30 to 100 of them
// deep, so copying match after match is a chain of waits.  Here the output
// goes by windows, and every byte of a window gets its distance back to the
// byte it copies (0: a literal).  Where that lies in the window too, the
// distance there is added, for all bytes at once, until none changes: each
// round doubles the links followed, so three to five rounds do.  Then each
// byte has its value before the window or in a literal, and one gather writes
// the window.  Distances may be read while others replace them: old or new,
// they lead to the same byte.  Four forms that copied matches instead (every
// match waiting for its own source; the late ones by one warp in order, or by
// all in rounds) took 185,000-260,000 cycles a short-read member.
//
// Distances past a window's end, of its last match, stay in the ring's other
// half for the next window.
template <int NW> __device__ void copy_matches(Smem<NW> *sm, u32 skew, u32 n)
{
    constexpr u32 NT = Smem<NW>::NT, WIN = Smem<NW>::WIN, PER = WIN / 2 / NT;
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid / 32;
    const u32 out = smem_u32(sm->out), list = smem_u32(sm->end) + (GROUP_MATCHES + 3u) * warp, marks = smem_u32(sm->starts);
    const u32 ring = smem_u32(sm->back), total = skew + n;
    for (u32 i = tid; i < WIN; i += NT) sts32(ring + 4u * i, 0);
    __syncthreads();
    bool reach = false;
    u32 zone = 0; // the ring's half of this window
    for (u32 window = 0; window < total; window += WIN, zone ^= WIN) {
        for (u32 rel = 256u * warp; rel < WIN && window + rel < total; rel += 256u * NW) {
            // a group's matches: a lane looks at the marks of eight bytes, at most three
            const u32 at = marks + (window + rel) / 8u + lane;
            u32 m = lds8(at);
            sts8(at, 0);
            const u32 c = __popc(m);
            const u32 c0 = __ballot_sync(FRT_FULL_MASK, c & 1u), c1 = __ballot_sync(FRT_FULL_MASK, c & 2u);
            const u32 to = list + __popc(c0 & lanemask_lt()) + 2u * __popc(c1 & lanemask_lt());
            const u32 count = __popc(c0) + 2u * __popc(c1);
#pragma unroll
            for (u32 k = 0; k < 3; ++k) {
                sts8_if(m != 0, to + k, 8u * lane + __ffs(m) - 1u);
                m &= m - 1;
            }
            __syncwarp();
            for (u32 k = lane; k < ((count + 31u) & ~31u); k += 32) {
                const bool on = k < count;
                const u32 r = rel + lds8_if(on, list + k), d = out + window + r, sh = 8u * (d & 3u);
                const u32 v = __funnelshift_r(lds32_if(on, d & ~3u), lds32_if(on && sh > 8u, (d & ~3u) + 4), sh) & 0xffffffu;
                const u32 dist = (v & 0x7fffu) + 1u, len = (v >> 15) + 3u;
                const bool bad = on && dist > window + r - skew;
                reach |= bad;
                // by a lane: up to 64 bytes, none of them its own source, all on this side of the ring's end
                const bool run = on && len <= 64u && len <= dist && zone + r + len <= 2u * WIN;
                u32 slot = ring + 2u * (zone + r), few = run && !bad ? len : 0u;
                do {
                    sts16_run(slot, few, dist);
                    slot += 16;
                    few = few > 8u ? few - 8u : 0u;
                } while (__any_sync(FRT_FULL_MASK, few));
                for (u32 b = __ballot_sync(FRT_FULL_MASK, on && !run && !bad); b; b &= b - 1) { // others by the warp
                    const u32 l = __ffs(b) - 1;
                    const u32 rr = __shfl_sync(FRT_FULL_MASK, zone + r, l), nn = __shfl_sync(FRT_FULL_MASK, len, l);
                    const u32 di = __shfl_sync(FRT_FULL_MASK, dist, l);
                    for (u32 i = lane; i < nn; i += 32) {
                        const u32 x = rr + i < 2u * WIN ? rr + i : rr + i - 2u * WIN;
                        sts16(ring + 2u * x, di < nn ? di + i - i % di : di);
                    }
                }
            }
            __syncwarp();
        }
        __syncthreads();
        // rounds: a thread has PER pairs of bytes
        u32 w[PER], live = 0; // two bits a pair: bytes whose distance may still grow
#pragma unroll
        for (u32 k = 0; k < PER; ++k) {
            const u32 rel = 2u * (tid + NT * k);
            w[k] = lds32(ring + 2u * (zone + rel));
            live |= ((w[k] & 0xffffu) - 1u < rel ? 1u : 0u) << (2 * k);
            live |= ((w[k] >> 16) - 1u < rel + 1u ? 2u : 0u) << (2 * k);
        }
        while (__syncthreads_or(live)) {
#pragma unroll
            for (u32 k = 0; k < PER; ++k) {
                if (!__any_sync(FRT_FULL_MASK, live & (3u << (2 * k)))) continue;
                const u32 rel = 2u * (tid + NT * k), at = ring + 2u * (zone + rel);
                const u32 a = lds16_if((live >> (2 * k)) & 1u, at - 2u * (w[k] & 0xffffu));
                const u32 b = lds16_if((live >> (2 * k)) & 2u, at + 2u - 2u * (w[k] >> 16));
                w[k] += a + (b << 16);
                sts32_if(a | b, at, w[k]);
                // a source of distance 0 is a literal; one before the window is final
                if (a == 0 || (w[k] & 0xffffu) - 1u >= rel) live &= ~(1u << (2 * k));
                if (b == 0 || (w[k] >> 16) - 1u >= rel + 1u) live &= ~(2u << (2 * k));
            }
        }
#pragma unroll
        for (u32 k = 0; k < PER; ++k) {
            const u32 rel = 2u * (tid + NT * k), at = out + window + rel;
            const u32 a = lds8_if(w[k] != 0, at - (w[k] & 0xffffu)), b = lds8_if(w[k] != 0, at + 1u - (w[k] >> 16));
            sts16_if(w[k] != 0, at, a | (b << 8));
            sts32(ring + 2u * (zone + rel), 0);
        }
        __syncthreads();
    }
    if (__syncthreads_or(reach) && tid == 0) sm->fail = 1;
    __syncthreads();
}

// CRC-32 of out[0, n) by the team.
template <int NW> __device__ u32 crc_of(Smem<NW> *sm, const u8 *out, u32 n)
{
    const u32 tid = threadIdx.x, NT = Smem<NW>::NT;
    if (tid == 0) sm->sh[7] = 0;
    for (u32 i = tid; i < 1024; i += NT) sm->crc[i >> 8][i & 255u] = g_crc.slice[i >> 8][i & 255u];
    __syncthreads();
    const u32 head = min(n, (4u - ((u32)(u64)out & 3u)) & 3u), nw = (n - head) / 4u;
    const u32 per = ((nw + NT - 1) / NT) | 1u; // words a thread: odd, so no bank conflicts
    const u32 w0 = min(nw, tid * per), w1 = min(nw, w0 + per);
    u32 c = 0;
    const u32 *words = (const u32 *)(out + head);
    if (tid == 0) {
        c = 0xffffffffu;
        for (u32 i = 0; i < head; ++i) c = sm->crc[0][(c ^ out[i]) & 0xffu] ^ (c >> 8);
    }
    for (u32 i = w0; i < w1; ++i) {
        c ^= words[i];
        c = sm->crc[3][c & 0xffu] ^ sm->crc[2][(c >> 8) & 0xffu] ^ sm->crc[1][(c >> 16) & 0xffu] ^ sm->crc[0][c >> 24];
    }
    u32 end = head + 4u * w1;
    if (w1 == nw && (w0 < nw || tid == 0)) { // the thread of the last word takes the bytes after it
        for (; end < n; ++end) c = sm->crc[0][(c ^ out[end]) & 0xffu] ^ (c >> 8);
    }
    const u32 after = n - end;
    if (c) {
        c = gf2_mulmod(g_crc.xpow[after & 4095u], c);
        if (after >> 12) c = gf2_mulmod(g_crc.xpow4k[after >> 12], c);
    }
    c = __reduce_xor_sync(FRT_FULL_MASK, c);
    __syncthreads();
    if ((tid & 31u) == 0) atomicXor(&sm->sh[7], c);
    __syncthreads();
    return ~sm->sh[7];
}

// Writes out[0, n) to its place: the two have the same address modulo 16.
template <int NW> __device__ void write_out(const u8 *out, u8 *to, u32 n)
{
    const u32 tid = threadIdx.x, NT = Smem<NW>::NT;
    const u32 head = min(n, (16u - ((u32)(u64)to & 15u)) & 15u), nv = (n - head) / 16u;
    if (tid < head) to[tid] = out[tid];
    const uint4 *a = (const uint4 *)(out + head);
    uint4 *b = (uint4 *)(to + head);
    for (u32 i = tid; i < nv; i += NT) b[i] = a[i];
    const u32 done = head + 16u * nv;
    if (tid < n - done) to[done + tid] = out[done + tid];
}

// The member's compressed words from bit `bitpos` on, as many as the stage
// holds (`skew`: the payload's first bit in its first word).  Returns the
// staged place of payload bit 0: staged bit = payload bit + this, modulo 2^32.
template <int NW>
__device__ __forceinline__ u32 stage_from(Smem<NW> *sm, const u32 *base, u32 words, u32 skew, u32 bitpos)
{
    const u32 w0 = (skew + bitpos) >> 5;
    __syncthreads(); // the words before are no longer read
    for (u32 i = threadIdx.x; i < STAGE_WORDS; i += Smem<NW>::NT) {
        if (w0 + i < words) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((u32)__cvta_generic_to_shared(sm->stage + i)), "l"(base + w0 + i) : "memory");
        } else {
            sm->stage[i] = 0;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    return skew - 32u * w0;
}

constexpr u32 REPAIRS = 6; // rounds of counting again before all starts may be tried (12 measured 0-20% slower, 8 5%)

// One segment from `start`, counted: its end, from `from` on, how it stopped and
// its output bytes.
__device__ __forceinline__ u32 count_segment(u32 stage, u32 tab, u32 off, u32 from, u32 to, u32 start)
{
    if (start >= to) return start - from;
    Walk k;
    k.start(stage, off + start);
    const u32 lim = off + to;
    u32 e, bytes = 0;
    do {
        e = k.step(tab);
        bytes += (e >> 18) & 511u;
    } while (!(e & 1u) && (k.a < lim || k.b4 != 0u));
    return (k.a - off - from) | ((e & 1u ? e & 3u : 0u) << 10) | (bytes << 12);
}

// Maps of a place to a place, sixteen to a word of nibbles; 15 stays 15.
__device__ __forceinline__ unsigned long long then(unsigned long long first, unsigned long long second, u32 places)
{
    unsigned long long m = 0;
    for (u32 d = 0; d < places; ++d) m |= ((second >> (4u * ((u32)(first >> (4u * d)) & 15u))) & 15ull) << (4u * d);
    return m | ~0ull << (4u * places);
}

// The lanes' starts where they do not fall into step (codes of nearly one
// length: 64 or 128 equally likely symbols).  Counting again proves one lane
// more a round there, 55 to 216 rounds for a member of 64 KiB.  But a segment
// begins within a code's length of its boundary, unless a match's extra bits
// reach over it: so each lane counts its segment from every such place, which
// maps the place to one in the next segment, and the maps, joined over a warp,
// take the chain through it in one step.  A warp with a lane that leads to
// none of the places is followed lane by lane, counting where it has to.
// Measured on 4,000 members of 64 KiB, inflate alone in ms, counting again only,
// with this, and the serial variant: 128 symbols, Huffman codes only 24.0, 5.1
// and 10.4, zlib level 6 19.0, 6.1 and 10.5; 64 symbols 16.2, 5.1 and 10.2, and
// at level 6, which finds too many matches for this, 6.1, 6.1 and 10.4.
//
// Leaves the last lane in sh[3], how it stopped in sh[0] and its end in sh[1];
// returns the lane's start and, above, its bytes.
template <int NW>
__device__ __noinline__ unsigned long long settle(Smem<NW> *sm, u32 off, u32 bitpos, u32 seg, u32 nl, u32 total)
{
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid / 32;
    const u32 tab = smem_u32(sm->tab), stage = smem_u32(sm->stage);
    const u32 from = bitpos + tid * seg, to = min(bitpos + (tid + 1) * seg, total);
    u32 places = 1; // as many as the literal/length codes have bits, but for the rarest 64th
    while (places < 15 && sm->lit.lim[places] < 32768u - 512u) ++places;
    u32 found[15];
    unsigned long long map = ~0ull << (4u * places);
    for (u32 d = 0; d < places; ++d) {
        u32 next = 15;
        if (tid < nl) {
            const u32 r = found[d] = count_segment(stage, tab, off, from, to, from + d);
            if (tid + 1 < nl && !(r >> 10 & 3u) && (r & 1023u) - seg < places) next = (r & 1023u) - seg;
        }
        map |= (unsigned long long)next << (4u * d);
    }
#pragma unroll
    for (u32 k = 1; k < 32; k <<= 1) {
        const unsigned long long before = __shfl_up_sync(FRT_FULL_MASK, map, k);
        if (lane >= k) map = then(before, map, places);
    }
    const unsigned long long through = __shfl_sync(FRT_FULL_MASK, map, 31), before = __shfl_up_sync(FRT_FULL_MASK, map, 1);
    if (tid == 0) {
        sm->sh[2] = bitpos;
        sm->sh[3] = ~0u;
    }
    u32 start = 0, bytes = 0;
    for (u32 w = 0; w < NW; ++w) {
        __syncthreads();
        if (warp != w || sm->sh[3] != ~0u) continue;
        u32 in = sm->sh[2];
        const u32 place = in - (bitpos + 32 * w * seg);
        if (place < places && (through >> (4u * place) & 15u) != 15u) {
            const u32 mine = lane ? (u32)(before >> (4u * place)) & 15u : place;
            start = from + mine;
            bytes = found[mine] >> 12;
            in = bitpos + 32 * (w + 1) * seg + ((u32)(through >> (4u * place)) & 15u);
        } else {
            for (u32 j = 0; j < 32; ++j) {
                u32 r = 0;
                if (lane == j) {
                    r = in - from < places ? found[in - from] : count_segment(stage, tab, off, from, to, in);
                    start = in;
                    bytes = r >> 12;
                }
                r = __shfl_sync(FRT_FULL_MASK, r, j);
                in = bitpos + (32 * w + j) * seg + (r & 1023u);
                if ((r >> 10 & 3u) || 32 * w + j == nl - 1) {
                    if (lane == 0) {
                        sm->sh[0] = r >> 10 & 3u;
                        sm->sh[1] = in;
                        sm->sh[3] = 32 * w + j;
                    }
                    break;
                }
            }
        }
        if (lane == 0) sm->sh[2] = in;
    }
    __syncthreads();
    return start | ((unsigned long long)bytes << 32);
}

// A block costs the team some 26 us (its tables, the staging, the barriers) and
// 0.5 us a kilobit, a warp of the serial form 21 and 15; a CTA has twelve of
// those, which slow each other down twofold.  So members of several short
// blocks are the serial form's, where enough of them are at hand: by BRIEF bits
// a block for each further member a CTA has, up to BRIEF_SHARE.  Measured on
// short-read members of 65,280 bytes by zlib's memLevel (bits a block), in ms
// the team alone, the serial variant, and the two as they are chosen:
//                  1,000 members       4,000               10,000
//   1  (1,200)   22.9  10.2   9.3    83.5  23.8  22.6    203   49.3  40.8
//   2  (2,400)   11.3   7.1   6.8    41.1  16.3  16.1    100   33.4  28.7
//   3  (4,800)    5.8   5.7   5.8    21.0  12.5  13.0     51.0 26.2  23.3
//   4  (9,600)    3.1   5.0   3.1    11.4  11.1  11.9     27.6 23.3  21.2
//   5 (19,000)    1.7   4.8   1.7     6.2  10.9   6.3     15.0 22.1  15.1
constexpr u32 BRIEF = 1500, BRIEF_SHARE = 7;

// One Huffman block from bit `bitpos` (its tables built): bitpos moves past
// its end-of-block code, pos over its bytes.  `off` is the staged place of bit
// 0 (stage_from), and moves with the stage.  False (uniform): the serial form is to take the member.
template <int NW>
__device__ __forceinline__ bool decode_block(Smem<NW> *sm, const u32 *base, u32 words, u32 skew, u32 total, u32 out_at,
                                             u32 cap, u32 &off, u32 &bitpos, u32 &pos, bool last_block)
{
    constexpr u32 NT = Smem<NW>::NT;
    constexpr u32 SYNC_BITS = 640, MIN_SEG = 192; // 512 and 768, 256 and 384 measured 0-4% slower
    const u32 block_at = bitpos;
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid / 32;
    const u32 tab = smem_u32(sm->tab), stage = smem_u32(sm->stage), out = smem_u32(sm->out), starts = smem_u32(sm->starts);
    while (true) {
        const u32 rem = total - bitpos;
        if (rem == 0) return false; // ends before the block does
        // the last block takes the rest of the payload, others about what the
        // one before took: a block that ends in its round takes one round, and
        // lanes past its end work for nothing
        const u32 guess = min(last_block ? rem : min(rem, sm->hint), ROUND_BITS - (off + bitpos));
        const u32 seg = max(MIN_SEG, (guess + NT - 1) / NT);
        const u32 nl = min(min(NT, (rem + seg - 1) / seg), max(1u, (ROUND_BITS - (off + bitpos)) / seg)); // lanes with a segment
        const u32 from = bitpos + tid * seg, to = min(bitpos + (tid + 1) * seg, total);
        const bool mine = tid < nl;
        u32 w = 0, start = bitpos, end = 0, bytes = 0, stop = 0;
        Walk k;
        if (mine && tid) { // 1. sync
            k.start(stage, off + (tid * seg <= SYNC_BITS ? bitpos : from - SYNC_BITS));
            const u32 lim = off + from;
            do k.step(tab);
            while (k.a < lim || k.b4 != 0u);
            start = k.a - off;
        }
        bool count = mine;
        u32 E, F, rounds = 0;
        while (true) { // 2. count
            if (count) {
                bytes = stop = 0;
                end = start;
                if (start < to) {
                    k.start(stage, off + start);
                    const u32 lim = off + to;
                    u32 e;
                    do {
                        e = k.step(tab);
                        bytes += (e >> 18) & 511u;
                    } while (!(e & 1u) && (k.a < lim || k.b4 != 0u));
                    stop = (e & 1u) ? (e & 3u) : 0u;
                    end = k.a - off;
                }
                sm->end[tid] = end;
            }
            __syncthreads();
            const u32 before = tid && mine ? sm->end[tid - 1] : bitpos;
            const bool apart = mine && start != before;
            const u32 so = __ballot_sync(FRT_FULL_MASK, mine && stop != 0), mo = __ballot_sync(FRT_FULL_MASK, apart);
            if (lane == 0) {
                sm->wa[warp] = so ? tid + __ffs(so) - 1u : 0xffffu;
                sm->wb[warp] = mo ? tid + __ffs(mo) - 1u : 0xffffu;
            }
            __syncthreads();
            E = __reduce_min_sync(FRT_FULL_MASK, lane < NW ? sm->wa[lane] : 0xffffu); // first lane that stopped
            F = __reduce_min_sync(FRT_FULL_MASK, lane < NW ? sm->wb[lane] : 0xffffu); // first lane out of step
            E = min(E, nl - 1u);
            if (F > E) break;
            // Starts by all places where many lanes are still apart (one in
            // eight, and 24: fewer are proven sooner) and next to none ends far over its boundary, in a match:
            // a warp with one that does takes settle as long as eight rounds.
            if (++rounds % REPAIRS == 0 && 8 * __syncthreads_count(apart) > max(nl, 192u) &&
                128 * __syncthreads_count(mine && stop == 0 && end - to >= 12u) < nl) {
                const unsigned long long r = settle<NW>(sm, off, bitpos, seg, nl, total);
                start = (u32)r;
                bytes = (u32)(r >> 32);
                E = sm->sh[3];
                stop = sm->sh[0];
                end = sm->sh[1];
                break;
            }
            count = apart && tid <= E;
            if (count) start = before;
        }
        // lanes 0..E hold the block's next symbols; their places in the output
        u32 a = tid <= E ? bytes : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const u32 x = __shfl_up_sync(FRT_FULL_MASK, a, d);
            if ((int)lane >= d) a += x;
        }
        __syncthreads();
        if (lane == 31) sm->wa[warp] = a;
        if (tid == E) {
            sm->sh[0] = stop;
            sm->sh[1] = end;
        }
        __syncthreads();
        const u32 wa = lane < NW ? sm->wa[lane] : 0u;
        a += __reduce_add_sync(FRT_FULL_MASK, lane < warp ? wa : 0u);
        const u32 tot = __reduce_add_sync(FRT_FULL_MASK, wa), how = sm->sh[0], next = sm->sh[1];
        if (how == F_BAD || next > total || (how == 0 && next >= total) || tot > cap - pos) return false;
        if (tid <= E && start < to) { // 3. emit
            // no branches but the loop's: stores are predicated, and what is
            // computed for the other kinds of code is dropped.  A code's
            // stores wait for the next one's lookups to be under way.
            u32 o = out_at + pos + a - bytes, ml = 0, e = 0, v = 0;
            k.start(stage, off + start);
            const u32 lim = off + to;
            bool more;
            do {
                const u32 w0 = w, e0 = e, v0 = v;
                e = k.step(tab, (u32)(offsetof(Smem<NW>, val) - offsetof(Smem<NW>, tab)), w, v);
                emit_code(out, starts, e0, v0, w0, o, ml);
                k.pass(e);
                more = !(e & 1u) && (k.a < lim || k.b4 != 0u);
            } while (more);
            emit_code(out, starts, e, v, w, o, ml);
        }
        bitpos = next;
        pos += tot;
        __syncthreads();
        if (how == F_END) {
            if (!last_block && tid == 0) sm->hint = bitpos - block_at + (bitpos - block_at) / 16u;
            return true;
        }
        off = stage_from<NW>(sm, base, words, skew, bitpos);
    }
}

// Inflates one member; every thread gets the result.  False: the serial form
// is to take it (nothing was written to HBM).
template <int NW>
__device__ bool member(Smem<NW> *sm, const u8 *in, u32 in_len, u8 *to, u32 cap, u32 *produced, u32 *crc_out)
{
    constexpr u32 NT = Smem<NW>::NT;
    const u32 tid = threadIdx.x;
    if (cap > OUT_MAX || in_len == 0 || in_len > (1u << 28)) return false;
    const u32 out_at = (u32)(u64)to & 15u;
    u8 *const out = sm->out + out_at;
    const u32 *base = (const u32 *)((u64)in & ~3ull);
    const u32 skew = 8u * (u32)((u64)in & 3ull), total = 8u * in_len;
    const u32 words = (skew + total + 31u) / 32u; // only words that hold payload are read
    u32 bitpos = 0, pos = 0, off = 0;
    bool coded = false; // the block before: a stored one leaves nothing to wait for
    if (tid == 0) sm->blocks = 0;
    while (true) {
        if (bitpos + 3 > total) return false;
        if (coded) {
            if (tid == 0) {
                const u32 blocks = ++sm->blocks;
                if (blocks >= 2 && bitpos < blocks * sm->brief && total - bitpos > 2 * sm->brief) sm->fail = 1;
            }
            __syncthreads();
            if (sm->fail) return false;
        }
        // the words staged do while they hold a stored block's header, or a coded
        // block like the last one (any header, and a few segments): staging anew
        // for each, and its barriers, made a short stored block 3 us
        if (bitpos == 0 || off + bitpos + 64u > ROUND_BITS ||
            ((bits_at(sm->stage, off + bitpos) & 6u) &&
             off + bitpos + max(min(total - bitpos, sm->hint), HEAD_BITS + 1024u) > ROUND_BITS))
            off = stage_from<NW>(sm, base, words, skew, bitpos);
        const u32 v = bits_at(sm->stage, off + bitpos);
        const bool fin = v & 1u;
        const u32 type = (v >> 1) & 3u;
        bitpos += 3;
        if (type == 3) return false;
        if (type == 0) {
            const u32 at = (bitpos + 7u) / 8u;
            if (at + 4 > in_len) return false;
            const u32 x = bits_at(sm->stage, off + 8u * at), len = x & 0xffffu;
            if (len != (~(x >> 16) & 0xffffu) || at + 4 + len > in_len || len > cap - pos) return false;
            // from the stage as far as it goes, the rest from HBM
            const u8 *src = in + at + 4, *near = (const u8 *)sm->stage + (off + 8u * (at + 4)) / 8u;
            const u32 have = min(len, (ROUND_BITS - (off + 8u * at)) / 8u - 4u);
            for (u32 i = tid; i < have; i += NT) out[pos + i] = near[i];
            for (u32 i = have + tid; i < len; i += NT) out[pos + i] = src[i];
            bitpos = 8u * (at + 4 + len);
            pos += len;
            coded = false;
            // more of them, up to the last, that lie in the stage whole: the same
            // by staged bits
            for (u32 a = off + bitpos; !fin && a + 96u <= ROUND_BITS;) {
                const u32 *w = sm->stage + (a >> 5), w0 = w[0], w1 = w[1], w2 = w[2];
                const u32 a2 = (a + 10u) & ~7u, sh = a2 - (a & ~31u);
                const u32 y = sh < 32u ? __funnelshift_r(w0, w1, sh) : __funnelshift_r(w1, w2, sh - 32u), n = y & 0xffffu;
                const u32 past = a2 + 32u + 8u * n;
                if ((__funnelshift_r(w0, w1, a) & 7u) || (y ^ (n << 16)) >> 16 != 0xffffu ||
                    past > min(ROUND_BITS, off + total) || n > cap - pos)
                    break;
                for (u32 i = tid; i < n; i += NT) out[pos + i] = ((const u8 *)sm->stage)[(a2 >> 3) + 4u + i];
                pos += n;
                a = past;
                bitpos = a - off;
            }
        } else {
            coded = true;
            u32 nlen = 288, ndist = 32;
            if (type == 2) {
                u32 a = off + bitpos;
                if (!read_lengths<NW>(sm, a, nlen, ndist)) return false;
                bitpos = a - off;
                if (bitpos > total) return false;
            } else {
                for (u32 s = tid; s < 320; s += NT) sm->lens[s] = s < 144 ? 8 : (s < 256 ? 9 : (s < 280 ? 7 : (s < 288 ? 8 : 5)));
                __syncthreads();
            }
            if (!build<NW>(sm, nlen, ndist)) return false;
            if (!decode_block<NW>(sm, base, words, skew, total, out_at, cap, off, bitpos, pos, fin)) return false;
        }
        if (fin) break;
    }
    __syncthreads();
    copy_matches<NW>(sm, out_at, pos);
    if (sm->fail) return false;
    *crc_out = crc_of<NW>(sm, out, pos);
    write_out<NW>(out, to, pos);
    *produced = pos;
    __syncthreads();
    return true;
}

template <int NW> __device__ __forceinline__ void clear_marks(Smem<NW> *sm)
{
    for (u32 i = threadIdx.x; i < MARKS; i += Smem<NW>::NT) sm->starts[i] = 0;
    if (threadIdx.x == 0) {
        sm->fail = 0;
        sm->hint = 180000; // bits of the next block: 16,383 symbols (zlib's default) of eleven bits
    }
}

template <int NW> __device__ __forceinline__ void setup(Smem<NW> *sm)
{
    const u32 tid = threadIdx.x, NT = Smem<NW>::NT;
    clear_marks<NW>(sm);
    for (u32 i = tid; i < EXTRA_CAP; i += NT) { // lengths with extra bits: 4 symbols of x bits each, x = 1..5
        u32 x = 1;
        while (i >= 4u * ((1u << (x + 1)) - 2u)) ++x;
        const u32 j = i - 4u * ((1u << x) - 2u);
        sm->tab[EXTRA_AT + i] = to_dist(x, ((4u + (j >> x)) << x) + 3u + (j & ((1u << x) - 1u)));
    }
    __syncthreads();
}

// A launch's members.
struct Job {
    const u8 *in;
    const u64 *in_off;
    const u32 *in_len;
    u8 *out;
    const u64 *out_off;
    const u32 *cap;
    const u32 *crc_expect; // null: the caller checks
    u32 *status, *produced, *crc;
    unsigned long long *block_err;
    // A member's result, by one thread: with crc_expect, checked against its
    // trailer as in k_inflate_persistent.
    __device__ __forceinline__ void put(u32 m, u32 st, u32 p, u32 c) const
    {
        status[m] = st;
        produced[m] = p;
        crc[m] = st == INF_OK ? c : 0u;
        if (!crc_expect) return;
        const unsigned long long code = st != INF_OK ? 5ull : (p != cap[m] ? 4ull : (c != crc_expect[m] ? 3ull : 0ull));
        if (code) atomicMin(block_err, ((unsigned long long)m << 8) | code);
    }
};

using Serial = Cfg<9, 7, 1024, 192>;

__device__ unsigned long long g_handed_over; // members the team form left to the serial form

// The `listed` members of sm->list by the serial form, a warp each, in the place
// of the output and the block's tables.
template <int NW> __device__ __noinline__ void run_listed(Smem<NW> *sm, const Job &job, u32 listed)
{
    static_assert(NW * sizeof(WarpSmem<Serial>) <= offsetof(Smem<NW>, tab) + 4 * EXTRA_AT, "the serial form's states leave the rest");
    __syncthreads(); // the list is whole, and nothing else in use
    const u32 warp = threadIdx.x / 32;
    if (warp < listed) {
        const u32 m = sm->list[warp];
        u32 p = 0, c = 0;
        const u32 st = inflate_member_warp<Serial>(job.in + job.in_off[m], job.in_len[m], job.out + job.out_off[m], job.cap[m],
                                                   (WarpSmem<Serial> *)sm->out + warp, &p, &c);
        if (lane_id() == 0) job.put(m, st, p, c);
    }
    __syncthreads();
    clear_marks<NW>(sm);
    if (threadIdx.x == 0) {
        sm->listed = 0;
        atomicAdd(&g_handed_over, (unsigned long long)listed);
    }
    __syncthreads();
}

constexpr u32 NONE = 0xffffffffu;

// The CTA's next member, or NONE; by one thread, which keeps its place in
// shared memory: registers held through a member's decode cost it 1%.
template <int NW>
__device__ __forceinline__ u32 next_member(Smem<NW> *sm, const u32 *order, u32 n, u32 *queue_head, u32 chunk)
{
    u32 q = sm->q, end = sm->q_end, m = NONE;
    while (m >= n) { // an order may hold members past the launch's
        if (q == end) {
            u32 step = chunk;
            if (!order && end == 0) {
                q = blockIdx.x;
                step = 1;
            } else if (!order && gridDim.x >= n) {
                q = n;
            } else if (q < n) {
                q = atomicAdd(queue_head, chunk) + (order ? 0u : gridDim.x);
            }
            end = q < n ? min(n, q + step) : q;
            if (q >= n) {
                m = NONE;
                break;
            }
        }
        m = order ? order[q] : q;
        ++q;
    }
    sm->q = q;
    sm->q_end = end;
    return m;
}

// A grid of CTAs that pull members from a queue (`order`, or in their order)
// through an atomic head, `chunk` a pop.  Where no order is given, a CTA's first
// member is its own, and the queue begins after those.  (An ordered launch may
// share the SMs with others, as the slices of a file on its way here do: a CTA
// that runs takes members in the place of those that do not yet.)
//
// A member the team does not take is the serial form's.  Where a CTA has
// several members to do, such members wait on a list until there is one for
// each warp (alone, one leaves eleven warps idle).  One that is alone on the
// list at the end is the team's as far as it goes.  Where there are members to
// fill every CTA's list, the next ones after two in a row are listed untried.
template <int NW, int PER_SM>
__global__ void __launch_bounds__(32 * NW, PER_SM)
k_persistent(const u8 *in, const u64 *in_off, const u32 *in_len, u8 *out, const u64 *out_off, const u32 *isize,
             const u32 *crc_expect, u32 *status, u32 *produced, u32 *crc, const u32 *order, const u64 *n_ptr, u64 n_cap,
             u64 out_capacity, u32 *queue_head, u32 chunk, unsigned long long *block_err)
{
    extern __shared__ __align__(16) unsigned char smem[];
    Smem<NW> *sm = (Smem<NW> *)smem;
    const u64 n64 = n_ptr ? *n_ptr : n_cap;
    const u32 n = (u32)(n64 < n_cap ? n64 : n_cap);
    if (chunk == 0) chunk = 1;
    const Job job{in, in_off, in_len, out, out_off, isize, crc_expect, status, produced, crc, block_err};
    setup<NW>(sm);
    if (threadIdx.x == 0) {
        sm->brief = n ? BRIEF * min((n - 1u) / gridDim.x, BRIEF_SHARE) : 0u;
        sm->listed = sm->q = sm->q_end = sm->streak = 0;
    }
    while (true) {
        if (threadIdx.x == 0) sm->sh[6] = next_member<NW>(sm, order, n, queue_head, chunk);
        __syncthreads();
        u32 m = sm->sh[6];
        if (m == NONE) {
            const u32 listed = sm->listed;
            m = sm->list[0];
            if (listed > 1) run_listed<NW>(sm, job, listed);
            if (listed != 1) break;
            __syncthreads();
            if (threadIdx.x == 0) sm->listed = sm->brief = sm->streak = 0;
        }
        __syncthreads();
        const u32 cap = isize[m], len = in_len[m];
        const u64 from = in_off[m], to = out_off[m];
        if (to + cap > out_capacity) { // sizes changed since the buffers were planned
            if (threadIdx.x == 0) job.put(m, INF_OUTPUT_OVERFLOW, 0, 0);
            continue;
        }
        u32 p = 0, c = 0;
        if ((sm->streak < 2 || n / NW < gridDim.x) && member<NW>(sm, in + from, len, out + to, cap, &p, &c)) {
            if (threadIdx.x == 0) {
                job.put(sm->sh[6] != NONE ? sm->sh[6] : sm->list[0], INF_OK, p, c);
                sm->streak = 0;
            }
            continue;
        }
        __syncthreads();
        clear_marks<NW>(sm); // of what the team decoded before it gave up
        if (threadIdx.x == 0) {
            sm->list[sm->listed++] = sm->sh[6] != NONE ? sm->sh[6] : sm->list[0];
            ++sm->streak;
        }
        __syncthreads();
        if (sm->listed == NW || !sm->brief) {
            run_listed<NW>(sm, job, sm->listed);
            if (threadIdx.x == 0) sm->streak = 1;
        }
    }
}

} // namespace team
