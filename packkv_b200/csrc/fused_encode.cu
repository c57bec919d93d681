// Single-pass encoder: fp16/bf16 K or V -> packed stream blocks, without a code matrix in HBM.
//
// Replaces, for the north-star pairing (K per-channel, V per-token), the reference's
// quant_ints (torch, utils/compute.py:84-112) + k/v_encode_cpu (C++ on the host,
// packkv_cuda_ext/src/{k,v}_encode_cpu.cpp); codes, parameters and block bytes are identical to
// the separate quantise + pack kernels.
//
// The stream format lays blocks back to back, so a block's byte offset is the sum of all earlier
// block sizes of its sequence.  Three forms:
//   one block: ONE launch, for calls of one token block per sequence (what leaves the residual in a decode
//            step; up to 8 heads, see one_block_ctas): a cluster of one CTA per head takes a sequence, and
//            they get their offsets from one another's sizes through distributed shared memory.
//   direct : ONE launch.  A CTA builds its blocks (consecutive in the stream) in shared memory, then
//            learns the offset of its first block from the CTAs before it in the sequence by a
//            decoupled look-back over a small status array (every CTA publishes the bytes of its own
//            blocks as soon as it knows them, so nobody waits for more than its neighbours' packing),
//            and writes the blocks to their final place.  CTAs take their position from a ticket
//            counter, so every CTA a look-back waits for has started; the wait is bounded all the same
//            and a CTA that gives up raises the timeout flag and writes nothing.
//            HBM traffic per element: 2 B read (the second read of a tile comes from L1/L2) + the
//            block bytes written once (~0.56 B at 4 bit).
//   slots  : three launches, no device-side waiting (more than 8 heads in the kernels
//            with per-token parameters, short launches of V in 128-token blocks, or on request): encode into
//            fixed-stride SLOTS in scratch memory with the size in block_info[blk][1]; per-sequence
//            exclusive scan (scan_sizes_kernel, pack.cu); one warp per block copies its slot to its
//            final offset.  The block bytes are written, read and written once more.
#include <cooperative_groups.h>
#include <cstdlib>
#include <string>

#include "common.cuh"
#include "launch.h"
#include "pack_dev.cuh"
#include "quant_dev.cuh"

namespace cg = cooperative_groups;

namespace pkv {

struct FusedArgs {
    const void* x; int64_t sb, sh, ss;      // (B, H, S, 128), strides in elements
    void* scale; void* zero;
    int param_blocks, first_block;          // K channel mode parameter layout
    int param_tokens, first_token;          // V token mode parameter layout
    uint8_t* slots; int slot_stride;        // scratch: one slot per block, sequence-major
    uint32_t* info; int64_t info_seq_stride; int first_cb;
    int batch, heads, tokens, cb, bits;
    float rel;
    unsigned* flags;
    const uint8_t* order;                   // optional (batch, tokens / order_block, order_block): source row of every stored row
    int order_block;                        // tokens per reorder block (divides cb)
    // direct form (status != nullptr): blocks go straight to the stream
    unsigned* ticket;                       // zero before the launch: CTAs take their place in (sequence, link) order from it
    unsigned long long* status;             // [batch][links], zero before the launch: (state << 32) | bytes; state 1: this link's
                                            // blocks, 2: everything up to and including this link
    int links;                              // CTAs per sequence
    uint8_t* stream; int64_t stream_seq_stride, capacity;
    unsigned* stream_bytes;                 // per sequence: bytes in the stream before (in) and after (out) the call
};

#ifdef PKV_DEBUG_CHAIN
__device__ unsigned long long g_chain_stats[4];   // look-back cycles, look-backs, CTA cycles, CTAs
#endif
constexpr unsigned kChainSpins = 1u << 24;  // polls of a look-back before it gives up (each sleeps ~50 ns and waits for a load)

// The CTA's place in the launch: ticket t -> (sequence, link).  All threads call; one barrier.
__device__ __forceinline__ void chain_place(const FusedArgs& a, unsigned* sh_word, int& b, int& link) {
    if (a.links == 1) {          // nothing before it in its sequence: no place to take, no status to publish
        b = (int)(blockIdx.x + gridDim.x * blockIdx.y);
        link = 0;
        return;
    }
    if (threadIdx.x == 0) *sh_word = atomicAdd(a.ticket, 1u);
    __syncthreads();
    // sequences take turns: the links of one sequence that are in flight at the same time are few, so a look-back
    // rarely meets a predecessor that is still packing
    const unsigned t = *sh_word;
    b = (int)(t % (unsigned)a.batch);
    link = (int)(t / (unsigned)a.batch);
}

// Byte offset, in sequence b's stream, of the first block of link `link`, whose blocks hold `total` bytes in all.
// Called by ONE warp.  Returns false if a predecessor never published (bounded wait ran out).
__device__ __forceinline__ bool chain_offset(const FusedArgs& a, int b, int link, unsigned total, unsigned& offset) {
    const int lane = lane_id();
    unsigned long long* st = a.status + (int64_t)b * a.links;
    const unsigned base0 = a.first_cb == 0 ? 0u : a.stream_bytes[b];
    unsigned excl = 0;
    bool ok = true;
#ifdef PKV_DEBUG_CHAIN   // measurement builds: cycles and polls spent in look-backs
    const long long t_begin = clock64();
#endif
    if (link == 0) {
        excl = base0;
    } else {
        if (lane == 0) *reinterpret_cast<volatile unsigned long long*>(st + link) = (1ull << 32) | total;
        int j = link - 1;
        unsigned spins = 0;
        while (true) {
            const int idx = j - lane;
            const unsigned long long v = idx >= 0 ? *reinterpret_cast<volatile unsigned long long*>(st + idx) : ((2ull << 32) | base0);
            // the nearest link that knows everything before it ends the search; the links between it and this one
            // must have published their own bytes
            const unsigned done = __ballot_sync(0xffffffffu, (v >> 32) == 2);
            const int k = done ? __ffs(done) - 1 : 31;
            if (__any_sync(0xffffffffu, lane <= k && (v >> 32) == 0)) {
                if (++spins > kChainSpins) { ok = false; break; }
                __nanosleep(50);
                continue;
            }
            unsigned part = lane <= k ? (unsigned)v : 0u;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
            excl += part;
            if (done) break;
            j -= 32;
        }
    }
#ifdef PKV_DEBUG_CHAIN
    if (lane == 0) {
        atomicAdd(&g_chain_stats[0], (unsigned long long)(clock64() - t_begin));
        atomicAdd(&g_chain_stats[1], 1ull);
    }
#endif
    // successors must not hang on a link that gave up: it publishes its own bytes on top of what it has
    if (lane == 0) {
        if (a.links > 1) *reinterpret_cast<volatile unsigned long long*>(st + link) = (2ull << 32) | (excl + total);
        if (link == a.links - 1) a.stream_bytes[b] = excl + total;
        if (!ok) atomicOr(a.flags, kFlagTimeout);
    }
    offset = excl;
    return ok;
}

// One warp copies a finished block from shared memory (16-byte aligned) to its place in the stream (even address).
__device__ __forceinline__ void store_block(uint8_t* dst, const uint8_t* stage, int size, int lane) {
    const int head = min((int)(0u - (unsigned)reinterpret_cast<uintptr_t>(dst)) & 15, size);   // bytes before the first aligned chunk, even
    const int nfull = (size - head) >> 4;
    // the halfwords before the first chunk (at most seven, lanes 0 ..) and behind the last one (at most seven, lanes 8 ..)
    {
        const int at = lane < 8 ? 2 * lane : head + 16 * nfull + 2 * (lane - 8);
        if (at < (lane < 8 ? head : lane < 16 ? size : 0)) *reinterpret_cast<uint16_t*>(dst + at) = *reinterpret_cast<const uint16_t*>(stage + at);
    }
    const unsigned sh = (unsigned)(head & 3) * 8;                      // 0 or 16: byte offset inside the first source word of a chunk
    const unsigned* p = reinterpret_cast<const unsigned*>(stage + (head & ~3)) + 4 * lane;
    uint4* d = reinterpret_cast<uint4*>(dst + head) + lane;
    for (int c = lane; c < nfull; c += 32, p += 128, d += 32) {
        // aligned 32-bit loads, realigned by funnel shifts (the fifth word counts only where sh is not 0: then it is inside the block)
        const unsigned w0 = p[0], w1 = p[1], w2 = p[2], w3 = p[3], w4 = sh ? p[4] : 0u;
        *d = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
    }
}

// Direct form, after every warp of the CTA has put the sizes of its blocks into sizes[0..n): warp 0 gets the
// CTA's offset, then warp w stores the blocks w, w + nwarps, ... (block j at stage_of(j)) and their table entries.
// info_first: table index of block 0 of this link.  All threads call.
template <typename StageOf>
__device__ __forceinline__ void chain_store(const FusedArgs& a, int b, int link, const unsigned* sizes, int n, unsigned* sh_word, int64_t info_first,
                                            int nwarps, StageOf stage_of) {
    const int lane = lane_id(), wic = threadIdx.x >> 5;
    __syncthreads();
    if (wic == 0) {
        unsigned total = 0;
        for (int j = 0; j < n; j++) total += sizes[j];
        unsigned off;
        const bool ok = chain_offset(a, b, link, total, off);
        if (lane == 0) *sh_word = ok ? off : 0xFFFFFFFFu;
    }
    __syncthreads();
    const unsigned base = *sh_word;
    if (base == 0xFFFFFFFFu) return;
    for (int j = wic; j < n; j += nwarps) {
        unsigned off = base;
        for (int i = 0; i < j; i++) off += sizes[i];
        const unsigned size = sizes[j];
        uint32_t* bi = a.info + ((int64_t)b * a.info_seq_stride + info_first + j) * 2;
        if (lane == 0) { bi[0] = off; bi[1] = size; }
        if ((int64_t)off + size > a.capacity) {
            if (lane == 0) atomicOr(a.flags, kFlagStreamOverflow);
            continue;
        }
        store_block(a.stream + (int64_t)b * a.stream_seq_stride + off, stage_of(j), (int)size, lane);
    }
}

// A V block that lies in PARTS segments (part i at part(i), its bytes in sizes[i]) to dst: the table of segment ends, then the segments.
template <int PARTS, typename Part>
__device__ __forceinline__ void store_parts(uint8_t* dst, const unsigned* sizes, int lane, Part part) {
    unsigned end = 0;
#pragma unroll
    for (int i = 0; i < PARTS; i++) {
        store_block(dst + 2 * PARTS + end, part(i), (int)sizes[i], lane);
        end += sizes[i];
        if (lane == 0) *reinterpret_cast<uint16_t*>(dst + 2 * i) = (uint16_t)end;
    }
}
template <int PARTS>
__device__ __forceinline__ unsigned parts_size(const unsigned* sizes) {
    unsigned size = 2 * PARTS;
#pragma unroll
    for (int i = 0; i < PARTS; i++) size += sizes[i];
    return size;
}

// chain_store for n <= 32 blocks that lie in PARTS segments each (see store_parts): segment i of block j at part(j, i).
template <int PARTS, typename Part>
__device__ __forceinline__ void chain_store_parts(const FusedArgs& a, int b, int link, const unsigned* sizes, int n, unsigned* sh_word, int64_t info_first,
                                                  int nwarps, Part part) {
    const int lane = lane_id(), wic = threadIdx.x >> 5;
    __syncthreads();
    const unsigned mine = lane < n ? parts_size<PARTS>(sizes + lane * PARTS) : 0u;      // lane: block
    const unsigned incl = warp_inclusive_sum(mine);
    if (wic == 0) {
        unsigned off;
        const bool ok = chain_offset(a, b, link, __shfl_sync(0xffffffffu, incl, 31), off);
        if (lane == 0) *sh_word = ok ? off : 0xFFFFFFFFu;
    }
    __syncthreads();
    const unsigned base = *sh_word;
    if (base == 0xFFFFFFFFu) return;
    for (int j = wic; j < n; j += nwarps) {
        const unsigned size = __shfl_sync(0xffffffffu, mine, j), off = base + __shfl_sync(0xffffffffu, incl, j) - size;
        uint32_t* bi = a.info + ((int64_t)b * a.info_seq_stride + info_first + j) * 2;
        if (lane == 0) { bi[0] = off; bi[1] = size; }
        if ((int64_t)off + size > a.capacity) {
            if (lane == 0) atomicOr(a.flags, kFlagStreamOverflow);
            continue;
        }
        store_parts<PARTS>(a.stream + (int64_t)b * a.stream_seq_stride + off, sizes + j * PARTS, lane, [&](int i) { return part(j, i); });
    }
}

__device__ __forceinline__ void store_slot(uint8_t* slot, const uint8_t* stage, int size, int lane) {
    // slot and stage are 16-byte aligned; the slot has room for the rounded-up size
    for (int i = 16 * lane; i < size; i += 512) *reinterpret_cast<uint4*>(slot + i) = *reinterpret_cast<const uint4*>(stage + i);
}

// ------------------------------------------------------------------------------------------ K
// One round of a K block: quantise 16 tokens x 4 channels per lane and pack them at `at`: minima, lengths, packs.  row(t) gives the
// lane's four elements of the round's token t.  Returns the round's bytes.
template <typename T, int BITS, typename Row>
__device__ __forceinline__ unsigned k_encode_round(Row row, const Quantiser<T, false>& q0, const Quantiser<T, false>& q1, const Quantiser<T, false>& q2,
                                                   const Quantiser<T, false>& q3, uint8_t* at, int lane, unsigned& over) {
    constexpr int LB = len_field_bits(BITS), kMin = 16 * BITS, kLen = 16 * LB;
    const int z0 = (int)q0.zero, z1 = (int)q1.zero, z2 = (int)q2.zero, z3 = (int)q3.zero;
    unsigned u[16];                                   // four channel codes per token, one byte each
    unsigned mnj[4] = {255u, 255u, 255u, 255u}, mxj[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int t = 0; t < 16; t++) {
        const uint2 raw = row(t);
        const T* e = reinterpret_cast<const T*>(&raw);
        const unsigned c0 = q0.template code_u8<false>(QT<T>::ld(e), z0), c1 = q1.template code_u8<false>(QT<T>::ld(e + 1), z1);
        const unsigned c2 = q2.template code_u8<false>(QT<T>::ld(e + 2), z2), c3 = q3.template code_u8<false>(QT<T>::ld(e + 3), z3);
        mnj[0] = min(mnj[0], c0); mxj[0] = max(mxj[0], c0);
        mnj[1] = min(mnj[1], c1); mxj[1] = max(mxj[1], c1);
        mnj[2] = min(mnj[2], c2); mxj[2] = max(mxj[2], c2);
        mnj[3] = min(mnj[3], c3); mxj[3] = max(mxj[3], c3);
        u[t] = c0 | (c1 << 8) | (c2 << 16) | (c3 << 24);
    }
    unsigned minword = 0, lenword = 0, lens4 = 0;
    int len[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        over |= mxj[j] >> BITS;
        len[j] = min(bit_length_u32(mxj[j] - mnj[j]), BITS);
        minword |= (mnj[j] & ((1u << BITS) - 1u)) << (j * BITS);
        lenword |= (unsigned)len[j] << (j * LB);
        lens4 |= (unsigned)len[j] << (8 * j);
    }
    store_lane_fields_w<4 * BITS>(at, lane, minword);
    store_lane_fields_w<4 * LB>(at + kMin, lane, lenword);
    const unsigned inc = warp_inclusive_sum(lens4);
    const unsigned tot = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned exc = inc - lens4;
    uint8_t* packs = at + kMin + kLen;
    unsigned before = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        // tokens 0..7 and 8..15 as two words of at most 32 bits: w = w * 2^len + code, then the
        // minimum is taken off all eight fields at once (min * (1 + 2^len + ... + 2^(7 len)))
        const unsigned step = 1u << len[j];
        unsigned wt = 0, wb = 0, ones = 0;
#pragma unroll
        for (int t = 0; t < 8; t++) {
            wt = wt * step + __byte_perm(u[t], 0, 0x4440 + j);
            wb = wb * step + __byte_perm(u[t + 8], 0, 0x4440 + j);
            ones = ones * step + 1u;
        }
        wt -= mnj[j] * ones;
        wb -= mnj[j] * ones;
        const uint64_t w = ((uint64_t)wt << (8 * len[j])) | wb;
        store_pack_smem(packs + 2 * (before + ((exc >> (8 * j)) & 0xFFu)), w, len[j]);
        before += (tot >> (8 * j)) & 0xFFu;
    }
    return kMin + kLen + 2 * before;
}

// A pack's len halfwords to shared memory (even address): four predicated stores, 13 instructions less than with branches
__device__ __forceinline__ void sts_pack(unsigned at, uint64_t w, int len) {
    const unsigned lo = (unsigned)w, hi = (unsigned)(w >> 32);
    asm volatile(
        "{ .reg .pred a, b, c, d; .reg .b16 l0, l1, h0, h1;\n"
        "mov.b32 {l0, l1}, %1; mov.b32 {h0, h1}, %2;\n"
        "setp.gt.s32 a, %3, 0; setp.gt.s32 b, %3, 1; setp.gt.s32 c, %3, 2; setp.gt.s32 d, %3, 3;\n"
        "@a st.shared.u16 [%0], l0; @b st.shared.u16 [%0+2], l1; @c st.shared.u16 [%0+4], h0; @d st.shared.u16 [%0+6], h1; }"
        ::"r"(at), "r"(lo), "r"(hi), "r"(len) : "memory");
}
// The lanes' words of W bits (8, 12 or 16) as a bit string at shared address at (even).  All 32 lanes call.
template <int W>
__device__ __forceinline__ void sts_lane_fields(unsigned at, int lane, unsigned word) {
    static_assert(W == 8 || W == 12 || W == 16, "header fields of four channels");
    if (W == 8) {
        asm volatile("st.shared.u8 [%0], %1;" ::"r"(at + lane), "r"(word) : "memory");
    } else if (W == 16) {
        sts16(at + 2 * lane, (unsigned short)word);
    } else {                                             // four lanes' words are three halfwords: lanes 0, 1, 2 of four store one each
        const unsigned next = __shfl_down_sync(0xffffffffu, word, 1);
        const int i = lane & 3;
        if (i < 3) sts16(at + 6 * (lane >> 2) + 2 * i, (unsigned short)((word >> (4 * i)) | (next << (12 - 4 * i))));
    }
}

// A pack's word from its four groups of four tokens, 4 len bits each, in 16-bit lanes: tokens 0 .. 3 above 4 .. 7 in za, 8 .. 11 above 12 .. 15 in
// zb; step4 = 2^(4 len).
__device__ __forceinline__ uint64_t join_lanes(unsigned za, unsigned zb, int len, unsigned step4) {
    const unsigned close = step4 - 65536u, wt = (za >> 16) * close + za, wb = (zb >> 16) * close + zb;   // upper lane * 2^(4 len) + lower lane
    const unsigned step8 = step4 * step4;                                                               // 2^(8 len), 0 for len 4
    return (uint64_t)__funnelshift_lc(wt, 0u, 8 * len) << 32 | (wt * step8 + wb);
}

// The packs of four channels from the codes of 16 tokens and their minima and maxima (two channels to a word, 16-bit lanes): lengths
// (one to a byte in lens4) and words (token 0 in the top bits).  codes(j, t): channel j's codes of tokens t and t + 4, t's above.
template <int BITS, typename Codes>
__device__ __forceinline__ void pack_words(Codes codes, unsigned mn01, unsigned mx01, unsigned mn23, unsigned mx23,
                                           int (&len)[4], unsigned& lens4, uint64_t (&w)[4]) {
    const unsigned d01 = mx01 - mn01, d23 = mx23 - mn23;     // lane-wise: no borrow, max >= min
    const unsigned dj[4] = {d01 & 0xFFFFu, d01 >> 16, d23 & 0xFFFFu, d23 >> 16};
    lens4 = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        len[j] = min(bit_length_u32(dj[j]), BITS);
        lens4 |= (unsigned)len[j] << (8 * j);
        // 16-bit lanes, four tokens each (tokens 0 .. 3 above 4 .. 7, 8 .. 11 above 12 .. 15): z = z * 2^len + code for two of them per
        // multiply-add, then the minimum is taken off all four fields at once (min * (1 + 2^len + ... + 2^(3 len))); modulo 2^32, so
        // that the codes may carry a common offset that the minimum carries too.
        // In the end a lane is below 2^16: four codes below 2^4 at steps of at most 2^4.  Against one multiply-add and one
        // extraction per code: 1.6 instead of 2.8 instructions per code.
        unsigned step = 1u << len[j];
        asm("" : "+r"(step));                             // a number, or the compiler makes a shift and an addition of every multiply-add
        unsigned za = codes(j, 0), zb = codes(j, 8);
#pragma unroll
        for (int t = 1; t < 4; t++) {
            za = za * step + codes(j, t);
            zb = zb * step + codes(j, t + 8);
        }
        const unsigned step2 = step * step, off = 0u - (step2 * step + step2) - step - 1u, both = __byte_perm(j < 2 ? mn01 : mn23, 0, j & 1 ? 0x3232 : 0x1010);
        za += both * off;
        zb += both * off;
        w[j] = join_lanes(za, zb, len[j], step2 * step2);
    }
}

// A round of a K block (16 tokens x 128 channels, four channels to a lane) at `at`: minima, lengths, packs.  Returns its bytes.
template <int BITS>
__device__ __forceinline__ unsigned k_store_round(unsigned at, int lane, unsigned minword, unsigned lenword, unsigned lens4, const int (&len)[4],
                                                  const uint64_t (&w)[4]) {
    constexpr int LB = len_field_bits(BITS), kMin = 16 * BITS, kLen = 16 * LB;
    sts_lane_fields<4 * BITS>(at, lane, minword);
    sts_lane_fields<4 * LB>(at + kMin, lane, lenword);
    const unsigned inc = warp_inclusive_sum(lens4);
    const unsigned tot = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned exc2 = (inc - lens4) << 1;            // bytes: at most 2 * 31 * 4
    unsigned packs = at + kMin + kLen;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        sts_pack(packs + __byte_perm(exc2, 0, 0x4440 + j), w[j], len[j]);
        packs += 2 * __byte_perm(tot, 0, 0x4440 + j);
    }
    return packs - at;
}

// The same from the codes, as pack_words takes them; min01, min23: the minima without an offset that the codes may carry
template <int BITS, typename Codes>
__device__ __forceinline__ unsigned k_pack_round(Codes codes, unsigned min01, unsigned min23, unsigned mn01, unsigned mx01, unsigned mn23, unsigned mx23, unsigned at,
                                                 int lane) {
    constexpr unsigned kMask = (1u << BITS) - 1u;
    unsigned lenword = 0, lens4;
    int len[4];
    uint64_t w[4];
    pack_words<BITS>(codes, mn01, mx01, mn23, mx23, len, lens4, w);
#pragma unroll
    for (int j = 0; j < 4; j++) lenword |= (unsigned)len[j] << (j * len_field_bits(BITS));
    const unsigned minword = (min01 & kMask) | ((min01 >> 16 & kMask) << BITS) | ((min23 & kMask) << (2 * BITS)) | ((min23 >> 16 & kMask) << (3 * BITS));
    return k_store_round<BITS>(at, lane, minword, lenword, lens4, len, w);
}

// The same round for blocks whose four quantisers are packable(): two channels per instruction
// from the conversion to the pack minimum / maximum (16-bit lanes), then one multiply-add per code
// into the pack words.
template <typename T>
struct PackedQuantisers {
    unsigned k01, k23;
    HalfQuotient<T> h01, h23;                         // used when every quantiser is in the half domain
    __device__ __forceinline__ PackedQuantisers(const Quantiser<T, false>& q0, const Quantiser<T, false>& q1, const Quantiser<T, false>& q2, const Quantiser<T, false>& q3)
        : k01(packed_code_bias(q0, q1)), k23(packed_code_bias(q2, q3)), h01(q0, q1), h23(q2, q3) {}
};
template <typename T, int BITS, bool HALF, typename Row>
__device__ __forceinline__ unsigned k_encode_round_packed(Row row, const Quantiser<T, false>& q0, const Quantiser<T, false>& q1, const Quantiser<T, false>& q2,
                                                          const Quantiser<T, false>& q3, const PackedQuantisers<T>& pq, unsigned at, int lane, unsigned& over) {
    unsigned c01[16], c23[16];                        // HALF: with their channels' bias, which pack_words takes off with the minimum
    unsigned mn01 = 0xFFFFFFFFu, mx01 = 0u, mn23 = 0xFFFFFFFFu, mx23 = 0u;
#pragma unroll
    for (int t = 0; t < 16; t++) {
        const uint2 raw = row(t);
        c01[t] = HALF ? pq.h01.raw(raw.x) : packed_codes<T>(raw.x, q0, q1, pq.k01);
        c23[t] = HALF ? pq.h23.raw(raw.y) : packed_codes<T>(raw.y, q2, q3, pq.k23);
        mn01 = min_u16x2(mn01, c01[t]); mx01 = max_u16x2(mx01, c01[t]);
        mn23 = min_u16x2(mn23, c23[t]); mx23 = max_u16x2(mx23, c23[t]);
    }
    const unsigned k01 = HALF ? pq.k01 : 0u, k23 = HALF ? pq.k23 : 0u, min01 = mn01 - k01, min23 = mn23 - k23;
    over |= min01 | min23 | (mx01 - k01) | (mx23 - k23);      // a code below zero leaves its lane too
    const auto codes = [&](int j, int t) {
        return j < 2 ? __byte_perm(c01[t + 4], c01[t], j & 1 ? 0x7632 : 0x5410) : __byte_perm(c23[t + 4], c23[t], j & 1 ? 0x7632 : 0x5410);
    };
    return k_pack_round<BITS>(codes, min01, min23, mn01, mx01, mn23, mx23, at, lane);
}

__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// rounds of one K block, appended to `stage` behind the table of round ends
// MODE 0: scalar conversion, 1: two elements per instruction in fp32, 2: in the element type
// ORDERED: stored row t of the block is source row ordp[t] (16-byte aligned table of the block's rows)
template <typename T, int BITS, int MODE, bool ORDERED>
__device__ __forceinline__ int k_encode_rounds(const T* x, int64_t ss, const uint8_t* ordp, const Quantiser<T, false>& q0, const Quantiser<T, false>& q1,
                                               const Quantiser<T, false>& q2, const Quantiser<T, false>& q3, const KGeom& g, uint8_t* stage, int lane, bool& bad) {
    const PackedQuantisers<T> pq(q0, q1, q2, q3);
    const uint64_t row_bytes = 2 * (uint64_t)ss;
    const unsigned stage_a = smem_addr(stage);
    int pos = g.head_bytes;
    unsigned over = 0;
    for (int r = 0; r < g.rounds; r++) {
        uint4 ob = make_uint4(0, 0, 0, 0);
        if (ORDERED) ob = __ldg(reinterpret_cast<const uint4*>(ordp + 16 * r));
        const unsigned ow[4] = {ob.x, ob.y, ob.z, ob.w};
        if (r + 1 < g.rounds) {                            // the next round's rows to L1 (both halves of one row to two lanes): 128-token blocks, of which
            // an SM holds 12, 124 -> 110 us for 134 M elements; 64-token blocks, 24 to an SM, 95.7 and 95.3
            const int at = ORDERED ? ordp[16 * (r + 1) + (lane >> 1)] : 16 * (r + 1) + (lane >> 1);
            prefetch_l1(reinterpret_cast<const uint8_t*>(x - 4 * lane) + (uint64_t)(unsigned)at * row_bytes + 128 * (lane & 1));
        }
        const auto row = [&](int t) {
            const int at = ORDERED ? (int)__byte_perm(ow[t >> 2], 0, 0x4440 + (t & 3)) : r * 16 + t;
            return __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const uint8_t*>(x) + (uint64_t)(unsigned)at * row_bytes));
        };
        pos += MODE == 0 ? k_encode_round<T, BITS>(row, q0, q1, q2, q3, stage + pos, lane, over)
                         : k_encode_round_packed<T, BITS, MODE == 2>(row, q0, q1, q2, q3, pq, stage_a + pos, lane, over);
        if (lane == 0) *reinterpret_cast<uint16_t*>(stage + 2 * r) = (uint16_t)(pos - g.head_bytes);
    }
    bad = bad || (MODE == 0 ? over : over & ~(((1u << BITS) - 1u) * 0x00010001u)) != 0;
    return pos;
}

// one warp per K block (cb tokens x 128 channels of one head); lane owns channels 4l..4l+3, the
// same ownership as the stream format, so per-channel statistics need no cross-lane step.
// CONTIG: token rows are 128 elements apart (a contiguous (B, H, S, 128) tensor), so every load of a
// round is the block pointer plus a constant
#ifndef PKV_K_WARPS
#define PKV_K_WARPS 4
#endif
constexpr int kKWarps = PKV_K_WARPS;   // warps (= consecutive blocks of a sequence's stream) per CTA of the channel-mode K kernel
constexpr int kKWarpsOne = 8;          // and when that many blocks are all there is of a sequence: one CTA then needs no look-back
template <typename T, bool CONTIG, int BITS, bool ORDERED, int NW>
__global__ void __launch_bounds__(NW * 32, 768 / (NW * 32)) k_fused_encode_kernel(FusedArgs a) {
    const int64_t ss = CONTIG ? 128 : a.ss;
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = lane_id(), wic = threadIdx.x >> 5;
    const int nctx = a.tokens / a.cb;
    const int64_t per_seq = (int64_t)nctx * a.heads;
    __shared__ unsigned sh_word, sh_sizes[NW];
    const bool direct = a.status != nullptr;
    int b, rem, link = 0;
    int64_t warp = 0;
    if (direct) {
        // the CTA's warps take NW consecutive blocks of one sequence's stream
        chain_place(a, &sh_word, b, link);
        rem = link * NW + wic;
    } else {
        warp = (int64_t)blockIdx.x * NW + wic;
        if (warp >= per_seq * a.batch) return;
        b = (int)(warp / per_seq);
        rem = (int)(warp % per_seq);
    }
    const bool active = rem < per_seq;
    const int cbi = active ? rem / a.heads : 0, h = active ? rem % a.heads : 0;
    const KGeom g(a.cb, BITS);
    const int slot_smem = (g.head_bytes + g.rounds * (g.min_bytes + g.len_bytes + 128 * 2 * BITS) + 15) & ~15;
    uint8_t* stage = smem + wic * slot_smem;
    const T* x = reinterpret_cast<const T*>(a.x) + (int64_t)b * a.sb + (int64_t)h * a.sh + (int64_t)cbi * a.cb * ss + 4 * lane;
    int pos = 0;
    bool bad = false;
    if (active) {

    // per-channel min / max over the block, two channels per instruction in the element type
    // (min/max of element-type values is exact, so the fp32 detour is not needed here)
    using T2 = typename QT<T>::T2;
    T2 lo01 = QT<T>::init2(INFINITY), lo23 = lo01, hi01 = QT<T>::init2(-INFINITY), hi23 = hi01;
#pragma unroll 16
    for (int t = a.cb - 1; t >= 0; t--) {             // the first rows last: the first round finds them in L1
        const uint2 raw = __ldg(reinterpret_cast<const uint2*>(x + (int64_t)t * ss));
        const T2 v01 = *reinterpret_cast<const T2*>(&raw.x), v23 = *reinterpret_cast<const T2*>(&raw.y);
        lo01 = QT<T>::min2(lo01, v01); hi01 = QT<T>::max2(hi01, v01);
        lo23 = QT<T>::min2(lo23, v23); hi23 = QT<T>::max2(hi23, v23);
    }
    const float lo[4] = {QT<T>::lo_f(lo01), QT<T>::hi_f(lo01), QT<T>::lo_f(lo23), QT<T>::hi_f(lo23)};
    const float hi[4] = {QT<T>::lo_f(hi01), QT<T>::hi_f(hi01), QT<T>::lo_f(hi23), QT<T>::hi_f(hi23)};
    const Quantiser<T, false> q0(lo[0], hi[0], a.rel), q1(lo[1], hi[1], a.rel), q2(lo[2], hi[2], a.rel), q3(lo[3], hi[3], a.rel);
    {
        const int64_t pi = (((int64_t)b * a.heads + h) * a.param_blocks + a.first_block + cbi) * 128 + 4 * lane;
        T sc[4] = {QT<T>::cvt(q0.scale), QT<T>::cvt(q1.scale), QT<T>::cvt(q2.scale), QT<T>::cvt(q3.scale)};
        T zr[4] = {QT<T>::cvt(q0.zero), QT<T>::cvt(q1.zero), QT<T>::cvt(q2.zero), QT<T>::cvt(q3.zero)};
        *reinterpret_cast<uint2*>(reinterpret_cast<T*>(a.scale) + pi) = *reinterpret_cast<const uint2*>(sc);
        *reinterpret_cast<uint2*>(reinterpret_cast<T*>(a.zero) + pi) = *reinterpret_cast<const uint2*>(zr);
    }
    bad = q0.degenerate() || q1.degenerate() || q2.degenerate() || q3.degenerate();
    const bool packable = __all_sync(0xffffffffu, q0.packable() && q1.packable() && q2.packable() && q3.packable());
    const bool half_ok = __all_sync(0xffffffffu, q0.half_domain() && q1.half_domain() && q2.half_domain() && q3.half_domain());
    // reordered blocks (order_block == cb here): the table of this block's rows
    const uint8_t* ordp = ORDERED ? a.order + ((int64_t)b * nctx + cbi) * a.cb : nullptr;
    if (half_ok) pos = k_encode_rounds<T, BITS, 2, ORDERED>(x, ss, ordp, q0, q1, q2, q3, g, stage, lane, bad);
    else if (packable) pos = k_encode_rounds<T, BITS, 1, ORDERED>(x, ss, ordp, q0, q1, q2, q3, g, stage, lane, bad);
    else pos = k_encode_rounds<T, BITS, 0, ORDERED>(x, ss, ordp, q0, q1, q2, q3, g, stage, lane, bad);
    __syncwarp();
    }   // active
    if (direct) {
        if (lane == 0) sh_sizes[wic] = (unsigned)pos;
        const int64_t left = per_seq - (int64_t)link * NW;
        chain_store(a, b, link, sh_sizes, (int)(left < NW ? left : NW), &sh_word,
                    (int64_t)a.first_cb * a.heads + (int64_t)link * NW, NW, [&](int j) { return smem + j * slot_smem; });
    } else {
        store_slot(a.slots + (int64_t)warp * a.slot_stride, stage, pos, lane);
        if (lane == 0) a.info[((int64_t)b * a.info_seq_stride + (int64_t)(a.first_cb + cbi) * a.heads + h) * 2 + 1] = (unsigned)pos;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags, kFlagCodeRange);
}

// ------------------------------------------------------------------------------------------ V
// one CTA per (sequence, token block): pass 1 computes the per-token parameters over all heads
// (half a warp per token); pass 2 gives each warp whole V blocks (cb tokens x 64 channels), in one of two ways (v_form says which):
//   registers  two packs of 16 tokens at a time: a lane quantises four channels of the 16 tokens of one pack, two channels to an instruction,
//              and forms their pack words in registers as K's rounds do; the words then change lanes through shared memory, so that
//              a store covers the adjacent packs of 32 channels as the stream has them.  Fewer instructions.
//   tile       codes of eight channels of a token to a lane (16-byte loads) go to a transposed tile in shared memory, whose rows the packing
//              stage reads, a channel to a lane; the block comes out whole.  Fewer registers (16 warps twice to an SM without spills), shorter
//              chains for a warp that is alone, and whole blocks for the scratch of the slots form.
// One-block launches use the tile.
//
// Tile of one V block in shared memory, transposed for the packing stage: one row of CB bytes per
// channel, made of 16-byte chunks (one per pack); chunk p of channel ch is stored at chunk position
// p ^ v_swz(ch) so that both the word stores of the quantising stage and the 16-byte row reads of the
// packing stage spread over the banks.  Inside a chunk, byte 4*r0 + k holds token r0 + 4*k of the
// pack: the quantising lane with r0 = lane >> 3 owns those four tokens.
template <int CB>
__device__ __forceinline__ int v_swz(int ch) { return ((ch >> 1) ^ (ch >> 3)) & (CB / 16 - 1); }

// Codes of the eight channels a lane holds of token `tok`, two to a word.
template <typename T, int CB, int MODE>     // MODE 0: scalar conversion, 1: two elements per instruction in fp32, 2: in the element type
__device__ __forceinline__ void v_quantise_row(const uint4& raw, const float4* prm, int tok, unsigned (&c)[4]) {
    const uint4* prmh = reinterpret_cast<const uint4*>(prm + CB);   // per token: r, -128*scale, r/128 (element-type pairs), code bias
    const unsigned rw[4] = {raw.x, raw.y, raw.z, raw.w};
    if (MODE == 2) {
        const uint4 ph = prmh[tok];
        HalfQuotient<T> hq;
        hq.r = *reinterpret_cast<const typename QT<T>::T2*>(&ph.x);
        hq.nsp = *reinterpret_cast<const typename QT<T>::T2*>(&ph.y);
        hq.rp = *reinterpret_cast<const typename QT<T>::T2*>(&ph.z);
        hq.kab = ph.w;
        hq.magic = QT<T>::dup((float)(QT<T>::kIntBits == 0x6600u ? 1536 : 192));
        hq.pre = QT<T>::dup(QT<T>::kPre);
#pragma unroll
        for (int i = 0; i < 4; i++) c[i] = hq.codes(rw[i]);
        return;
    }
    const float4 pr = prm[tok];                            // scale, zero, 1/scale
    Quantiser<T, false> qz;
    qz.scale = pr.x; qz.zero = pr.y; qz.rcp = pr.z;
    if (MODE == 1) {
        const unsigned kab = __float_as_uint(pr.w);
#pragma unroll
        for (int i = 0; i < 4; i++) c[i] = packed_codes<T>(rw[i], qz, qz, kab);
    } else {
        const int zi = (int)pr.y;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 f = QT<T>::to_float2(rw[i]);
            c[i] = qz.template code_u8<false>(f.x, zi) | (qz.template code_u8<false>(f.y, zi) << 16);
        }
    }
}

// A lane's place in the tile of 64 channels: lane (r0 = lane >> 3, cg = lane & 7) turns its 4 tokens x 8 channels of a pack into one
// 4-token word per channel.
template <int CB>
struct TileLane {
    uint8_t* wr[4];                                        // row of channel 8cg + 2i at this lane's word, before the chunk swizzle
    int sw[4];
    __device__ __forceinline__ TileLane(uint8_t* tile, int lane) {
        const int r0 = lane >> 3, cg = lane & 7;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            wr[i] = tile + (8 * cg + 2 * i) * CB + 4 * r0;
            sw[i] = v_swz<CB>(8 * cg + 2 * i) << 4;       // channels 8cg + 2i and + 1 share the swizzle
        }
    }
    __device__ __forceinline__ void store(int p, const unsigned (&c)[4][4]) const {   // [token k][channel pair i] as 16-bit lanes
#pragma unroll
        for (int i = 0; i < 4; i++) {
            // (even channel | odd channel) x tokens 0..3 -> one word per channel
            const unsigned x = __byte_perm(c[0][i], c[1][i], 0x6240), y = __byte_perm(c[2][i], c[3][i], 0x6240);
            uint8_t* at = wr[i] + ((p << 4) ^ sw[i]);
            *reinterpret_cast<unsigned*>(at) = __byte_perm(x, y, 0x5410);
            *reinterpret_cast<unsigned*>(at + CB) = __byte_perm(x, y, 0x7632);
        }
    }
};

// Quantises one V block into the tile.  Lane (r0 = lane >> 3, cg = lane & 7) loads 8 channels
// (16 bytes) of tokens r0, r0+4, r0+8, ...
// Returns the OR of all codes in 16-bit lanes for the range check.
template <typename T, int CB, int MODE>
__device__ __forceinline__ unsigned v_quantise_tile(const T* src, int64_t ss, const float4* prm, const uint8_t* ord, uint8_t* tile, int lane) {
    const int r0 = lane >> 3;
    unsigned seen = 0;
    const TileLane<CB> out(tile, lane);
    const T* lsrc = src + 8 * (lane & 7);
#pragma unroll 1
    for (int p = 0; p < CB / 16; p++) {
        unsigned c[4][4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int tok = 16 * p + 4 * k + r0;
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(lsrc + (int64_t)ord[tok] * ss));
            v_quantise_row<T, CB, MODE>(raw, prm, tok, c[k]);
#pragma unroll
            for (int i = 0; i < 4; i++) seen |= c[k][i];
        }
        out.store(p, c);
    }
    return seen;
}

// One 16-byte tile chunk (word r0: bytes k = codes of tokens r0 + 4k of the pack) -> the pack's
// minimum, bit length and 2*len-byte word (token 0 in the top bits).
template <int BITS>
__device__ __forceinline__ void chunk_to_pack(const uint4& cw, int& len, uint64_t& wd, unsigned& mn1) {
    const unsigned wv[4] = {cw.x, cw.y, cw.z, cw.w};
    unsigned mn = 0xFFFFFFFFu, mx = 0u;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const unsigned ev = wv[i] & 0x00FF00FFu, od = (wv[i] >> 8) & 0x00FF00FFu;
        mn = min_u16x2(mn, min_u16x2(ev, od));
        mx = max_u16x2(mx, max_u16x2(ev, od));
    }
    mn1 = min(mn & 0xFFFFu, mn >> 16);
    const unsigned mx1 = max(mx & 0xFFFFu, mx >> 16);
    len = min(bit_length_u32(mx1 - mn1), BITS);
    unsigned step = 1u << len;
    asm("" : "+r"(step));                                 // see pack_words
    const unsigned rep = mn1 * 0x01010101u, step2 = step * step;
    // 16-bit lanes: tokens 0..3 above 4..7, 8..11 above 12..15, by Horner steps over the words (r0 = 0 highest)
    unsigned za = 0, zb = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const unsigned v = wv[i] - rep;
        za = za * step + __byte_perm(v, 0, 0x4041);
        zb = zb * step + __byte_perm(v, 0, 0x4243);
    }
    wd = join_lanes(za, zb, len, step2 * step2);
}

// One segment of a V block (PPT packs of 16 tokens for each of 32 channels) from the tile: this lane's channel row and swizzle.
// Minima, lengths, packs at `at`; returns the segment's bytes.
template <int CB, int BITS>
__device__ __forceinline__ unsigned v_pack_segment(const uint8_t* row, int swz, int r, uint8_t* at, int lane) {
    constexpr int LB = len_field_bits(BITS), PPT = CB == 32 ? 2 : 4, kMin = BITS * PPT * 4, kLen = LB * PPT * 4;
    unsigned minword = 0, lenword = 0, lens4 = 0;
    uint64_t wd[4];
    int len[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        len[q] = 0; wd[q] = 0;
        if (q < PPT) {
            // word r0 of the chunk: bytes k = tokens r0 + 4k of the pack
            const uint4 cw = *reinterpret_cast<const uint4*>(row + (((r * PPT + q) ^ swz) << 4));
            unsigned mn1;
            chunk_to_pack<BITS>(cw, len[q], wd[q], mn1);
            minword |= (mn1 & ((1u << BITS) - 1u)) << (q * BITS);
            lenword |= (unsigned)len[q] << (q * LB);
            lens4 |= (unsigned)len[q] << (8 * q);
        }
    }
    store_lane_fields_w<PPT * BITS>(at, lane, minword);
    store_lane_fields_w<PPT * LB>(at + kMin, lane, lenword);
    const unsigned inc = warp_inclusive_sum(lens4);
    const unsigned tot = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned exc = inc - lens4;
    const unsigned packs = smem_addr(at) + kMin + kLen;
    unsigned before = 0;
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (q < PPT) {
            sts_pack(packs + 2 * (before + ((exc >> (8 * q)) & 0xFFu)), wd[q], len[q]);
            before += (tot >> (8 * q)) & 0xFFu;
        }
    return kMin + kLen + 2 * before;
}

// One round (16 tokens x 128 channels) of a K block with per-token parameters from the two tiles of 64 channels
template <int CB, int BITS>
__device__ __forceinline__ unsigned kt_pack_round(const uint8_t* ctile, int r, uint8_t* at, int lane) {
    constexpr int LB = len_field_bits(BITS);
    unsigned minword = 0, lenword = 0, lens4 = 0;
    uint64_t wd[4];
    int len[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int ch = 4 * lane + j;                       // this lane's channel row and its chunk swizzle
        const uint8_t* row = ctile + (ch >> 6) * 64 * CB + (ch & 63) * CB;
        const uint4 cw = *reinterpret_cast<const uint4*>(row + ((r ^ v_swz<CB>(ch & 63)) << 4));
        unsigned mn1;
        chunk_to_pack<BITS>(cw, len[j], wd[j], mn1);
        minword |= (mn1 & ((1u << BITS) - 1u)) << (j * BITS);
        lenword |= (unsigned)len[j] << (j * LB);
        lens4 |= (unsigned)len[j] << (8 * j);
    }
    return k_store_round<BITS>(smem_addr(at), lane, minword, lenword, lens4, len, wd);
}

// What token_params_pass and the one-block kernel keep per token of one block
template <typename T, int CB>
__device__ __forceinline__ void put_token_params(const Quantiser<T, false>& qz, float4* prm, int t) {
    prm[t] = make_float4(qz.scale, qz.zero, qz.rcp, __uint_as_float(qz.packable() ? packed_code_bias(qz, qz) : 0u));   // bias 0 = not packable
    const HalfQuotient<T> hq(qz, qz);
    reinterpret_cast<uint4*>(prm + CB)[t] = make_uint4(*reinterpret_cast<const unsigned*>(&hq.r), *reinterpret_cast<const unsigned*>(&hq.nsp),
                                                       *reinterpret_cast<const unsigned*>(&hq.rp), qz.half_domain() ? hq.kab : 0u);
}

// Per-token quantisation parameters of one token block over all heads and channels (the
// reference's token mode reduces over dims [1, 4], utils/compute.py:405-410): half a warp per token takes its minimum and
// maximum, then thread t forms token t's parameters.  Writes (scale, zero, 1/scale, packed code bias or 0) to prm[] and, with WRITE, scale /
// zero to the caller's arrays; ord[t] = source row (inside the block) of stored row t.  One CTA barrier inside; the caller's next one must come
// before prm[] is read.  (Parameters formed by the half warp, every lane alike: 400 of a warp's 4700 instructions per block of 64 tokens x 8 heads.)
struct TokenState { bool bad, packed, half; };           // of this thread's token: degenerate; parameters that the two faster conversions take
template <typename T, int CB, bool WRITE = true, int NW = 8, bool FOURS = true>
__device__ __forceinline__ TokenState token_params_pass(const FusedArgs& a, const T* xb, float4* prm, const uint8_t* ord, int b, int cbi, int lane, int wic) {
    using T2 = typename QT<T>::T2;
    static_assert(NW * 32 >= CB, "a thread to a token");
    const auto min_of = [](unsigned x, unsigned y) {
        const T2 m = QT<T>::min2(*reinterpret_cast<const T2*>(&x), *reinterpret_cast<const T2*>(&y));
        return *reinterpret_cast<const unsigned*>(&m);
    };
    for (int t = 2 * wic + (lane >> 4); t < CB; t += 2 * NW) {     // 8 channels per lane
        const uint8_t* xt = reinterpret_cast<const uint8_t*>(xb + 8 * (lane & 15)) + (uint64_t)ord[t] * (2 * (uint64_t)a.ss);
        T2 lo2 = QT<T>::init2(INFINITY), hi2 = QT<T>::init2(-INFINITY);
        // eight heads' loads in flight together, with FOURS four where no more are left (eight of a single head: V 3 to 7 %, per-token K 4 % slower, 20 to 4096
        // CTAs; but V of 8 heads x 64 tokens, three CTAs of 8 warps to an SM, 16384 of them, takes 800 us with the second copy of the loads and 795 without)
        const auto take = [&](int h0, auto count) {
            constexpr int N = decltype(count)::value;
            uint4 raw[N];
#pragma unroll
            for (int i = 0; i < N; i++) {
                if (i == 0 || h0 + i < a.heads) raw[i] = __ldg(reinterpret_cast<const uint4*>(xt + (uint64_t)(unsigned)(h0 + i) * (2 * (uint64_t)a.sh)));
                else raw[i] = raw[0];
            }
#pragma unroll
            for (int i = 0; i < N; i++) {
                const T2 v0 = *reinterpret_cast<const T2*>(&raw[i].x), v1 = *reinterpret_cast<const T2*>(&raw[i].y);
                const T2 v2 = *reinterpret_cast<const T2*>(&raw[i].z), v3 = *reinterpret_cast<const T2*>(&raw[i].w);
                lo2 = QT<T>::min2(lo2, QT<T>::min2(QT<T>::min2(v0, v1), QT<T>::min2(v2, v3)));
                hi2 = QT<T>::max2(hi2, QT<T>::max2(QT<T>::max2(v0, v1), QT<T>::max2(v2, v3)));
            }
        };
        int h0 = 0;
        for (; a.heads - h0 > (FOURS ? 4 : 0); h0 += 8) take(h0, std::integral_constant<int, 8>{});
        if (FOURS && h0 < a.heads) take(h0, std::integral_constant<int, 4>{});
        // (minimum, -maximum) of the lane, then of the token: one minimum serves both
        const unsigned l = *reinterpret_cast<const unsigned*>(&lo2), u = *reinterpret_cast<const unsigned*>(&hi2) ^ 0x80008000u;
        unsigned m = min_of(__byte_perm(l, u, 0x5410), __byte_perm(l, u, 0x7632));
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) m = min_of(m, __shfl_xor_sync(0xffffffffu, m, s));
        if ((lane & 15) == 0) prm[t].x = __uint_as_float(m);
    }
    __syncthreads();
    const int t = threadIdx.x;
    if (t >= CB) return TokenState{false, true, true};
    const unsigned m = __float_as_uint(prm[t].x);
    const T2 both = *reinterpret_cast<const T2*>(&m);
    const Quantiser<T, false> qz(QT<T>::lo_f(both), -QT<T>::hi_f(both), a.rel);
    put_token_params<T, CB>(qz, prm, t);
    if (WRITE) {
        const int64_t pi = (int64_t)b * a.param_tokens + a.first_token + cbi * CB + t;
        reinterpret_cast<T*>(a.scale)[pi] = QT<T>::cvt(qz.scale);
        reinterpret_cast<T*>(a.zero)[pi] = QT<T>::cvt(qz.zero);
    }
    // (half_domain() implies packable(); a bias of 0 marks parameters that are not)
    return TokenState{qz.degenerate(), __float_as_uint(prm[t].w) != 0u, reinterpret_cast<const uint4*>(prm + CB)[t].w != 0u};
}

// Codes of a lane's four channels (at src) of the 16 tokens from tok0 on, with the tokens' parameters prm[], and their minima and maxima
// in 16-bit lanes.  ord: source row of every stored row (16-byte aligned).  The codes are kept as bytes, a word for two channels of
// tokens t and t + 4 (16 registers; with 16-bit lanes, 32 of them, the V kernel spills).
struct PackCodes {
    unsigned c01[8], c23[8], mn01, mx01, mn23, mx23;               // word 4 (t / 8) + t % 4: (t, t + 4) of the even channel, then of the odd one
    unsigned largest;                                              // OR of the maxima, before a code that is no byte (an error) lost its upper bits
    __device__ __forceinline__ unsigned operator()(int j, int t) const {
        const int at = 4 * (t >> 3) + (t & 3);
        return j < 2 ? __byte_perm(c01[at], 0, j & 1 ? 0x4243 : 0x4041) : __byte_perm(c23[at], 0, j & 1 ? 0x4243 : 0x4041);
    }
};
template <typename T, int CB, int MODE>     // MODE 0: scalar conversion, 1: two elements per instruction in fp32, 2: in the element type
__device__ __forceinline__ void quantise_pack(const uint8_t* src, uint64_t row_bytes, const float4* prm, const uint8_t* ord, int tok0, PackCodes& p) {
    const uint4* prmh = reinterpret_cast<const uint4*>(prm + CB);   // per token: r, -128*scale, r/128 (element-type pairs), code bias
    const uint4 ob = *reinterpret_cast<const uint4*>(ord + tok0);
    const unsigned ow[4] = {ob.x, ob.y, ob.z, ob.w};
    p.mn01 = 0xFFFFFFFFu; p.mx01 = 0u; p.mn23 = 0xFFFFFFFFu; p.mx23 = 0u;
    uint2 raw[16];
#pragma unroll
    for (int t = 0; t < 16; t++) raw[t] = __ldg(reinterpret_cast<const uint2*>(src + (uint64_t)__byte_perm(ow[t >> 2], 0, 0x4440 + (t & 3)) * row_bytes));
#pragma unroll
    for (int at = 0; at < 8; at++) {
        unsigned c[2][2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int t = 8 * (at >> 2) + (at & 3) + 4 * e;
            if (MODE == 2) {
                const uint4 ph = prmh[tok0 + t];
                HalfQuotient<T> hq;
                hq.r = *reinterpret_cast<const typename QT<T>::T2*>(&ph.x);
                hq.nsp = *reinterpret_cast<const typename QT<T>::T2*>(&ph.y);
                hq.rp = *reinterpret_cast<const typename QT<T>::T2*>(&ph.z);
                hq.kab = ph.w;
                hq.magic = QT<T>::dup((float)(QT<T>::kIntBits == 0x6600u ? 1536 : 192));
                hq.pre = QT<T>::dup(QT<T>::kPre);
                c[e][0] = hq.codes(raw[t].x);
                c[e][1] = hq.codes(raw[t].y);
            } else {
                const float4 pr = prm[tok0 + t];                    // scale, zero, 1/scale, packed code bias
                Quantiser<T, false> qz;
                qz.scale = pr.x; qz.zero = pr.y; qz.rcp = pr.z;
                if (MODE == 1) {
                    c[e][0] = packed_codes<T>(raw[t].x, qz, qz, __float_as_uint(pr.w));
                    c[e][1] = packed_codes<T>(raw[t].y, qz, qz, __float_as_uint(pr.w));
                } else {
                    const int zi = (int)pr.y;
                    const float2 f01 = QT<T>::to_float2(raw[t].x), f23 = QT<T>::to_float2(raw[t].y);
                    c[e][0] = qz.template code_u8<false>(f01.x, zi) | (qz.template code_u8<false>(f01.y, zi) << 16);
                    c[e][1] = qz.template code_u8<false>(f23.x, zi) | (qz.template code_u8<false>(f23.y, zi) << 16);
                }
            }
            p.mn01 = min_u16x2(p.mn01, c[e][0]); p.mx01 = max_u16x2(p.mx01, c[e][0]);
            p.mn23 = min_u16x2(p.mn23, c[e][1]); p.mx23 = max_u16x2(p.mx23, c[e][1]);
        }
        p.c01[at] = __byte_perm(c[0][0], c[1][0], 0x6240);
        p.c23[at] = __byte_perm(c[0][1], c[1][1], 0x6240);
    }
    p.largest = p.mx01 | p.mx23;
    if (p.largest & 0xFF00FF00u) {                                 // reported by the caller; the bytes are those of every form of the encoder
        p.mn01 = 0xFFFFFFFFu; p.mx01 = 0u; p.mn23 = 0xFFFFFFFFu; p.mx23 = 0u;
#pragma unroll
        for (int at = 0; at < 8; at++) {
            const unsigned e01 = __byte_perm(p.c01[at], 0, 0x4240), o01 = __byte_perm(p.c01[at], 0, 0x4341);
            const unsigned e23 = __byte_perm(p.c23[at], 0, 0x4240), o23 = __byte_perm(p.c23[at], 0, 0x4341);
            p.mn01 = min_u16x2(p.mn01, min_u16x2(e01, o01)); p.mx01 = max_u16x2(p.mx01, max_u16x2(e01, o01));
            p.mn23 = min_u16x2(p.mn23, min_u16x2(e23, o23)); p.mx23 = max_u16x2(p.mx23, max_u16x2(e23, o23));
        }
    }
}

// Four fields of W bits (the 16-bit lanes of f01, f23) as W / 2 bytes at `at` (even; 4-byte aligned for W = 8 and 16): the fields of
// four adjacent channels in a segment's header.
template <int W>
__device__ __forceinline__ void put_fields(uint8_t* at, unsigned f01, unsigned f23) {
    static_assert(W == 4 || W == 6 || W == 8 || W == 12 || W == 16, "header fields of one channel");
    const unsigned lo = W == 16 ? f01 : (f01 & 0xFFFFu) | (f01 >> 16 << W), hi = W == 16 ? f23 : (f23 & 0xFFFFu) | (f23 >> 16 << W);
    if (W == 16) {
        reinterpret_cast<unsigned*>(at)[0] = lo; reinterpret_cast<unsigned*>(at)[1] = hi;
    } else if (W == 12) {
        uint16_t* h = reinterpret_cast<uint16_t*>(at);
        h[0] = (uint16_t)lo; h[1] = (uint16_t)((lo >> 16) | (hi << 8)); h[2] = (uint16_t)(hi >> 8);
    } else if (W == 8) {
        *reinterpret_cast<unsigned*>(at) = lo | (hi << 16);
    } else if (W == 6) {
        const unsigned v = lo | (hi << 12);
        at[0] = (uint8_t)v; at[1] = (uint8_t)(v >> 8); at[2] = (uint8_t)(v >> 16);
    } else {
        *reinterpret_cast<uint16_t*>(at) = (uint16_t)(lo | (hi << 8));
    }
}

template <int CB, int BITS> struct VSegment {
    static constexpr int kPacks = CB == 32 ? 2 : 4, kGroups = CB == 128 ? 2 : 1, kCount = 2 * kGroups;   // packs per channel; 64-token groups; segments
    static constexpr int kMin = BITS * kPacks * 4, kLen = len_field_bits(BITS) * kPacks * 4, kBytes = kMin + kLen + 64 * kPacks * BITS, kBound = (kBytes + 15) & ~15;
};

// One V block (CB tokens x 64 channels at src) into its segments: segment i at stage + i * kBound, its bytes in sizes[i].
// Lane (par = lane >> 4, cg = lane & 15) takes channels 4cg .. 4cg + 3 of every other pack.  xch: 1280 bytes of the warp's, 16-byte aligned, in
// which the words change lanes.  A round takes about 670 instructions for a lane's 64 elements.  Returns the OR of the packs' largest codes in 16-bit lanes.
template <typename T, int CB, int BITS, int MODE>
__device__ __forceinline__ unsigned v_block_segments(const T* src, uint64_t row_bytes, const float4* prm, const uint8_t* ord, uint8_t* stage, uint8_t* xch, unsigned* sizes,
                                                     int lane) {
    using S = VSegment<CB, BITS>;
    constexpr int LB = len_field_bits(BITS);
    const int par = lane >> 4, cg = lane & 15, w = cg >> 3;
    const uint8_t* lsrc = reinterpret_cast<const uint8_t*>(src + 4 * cg);
    const unsigned stage_a = smem_addr(stage);
    uint2* words = reinterpret_cast<uint2*>(xch);                 // [128] pack words: pack 4 * lane + j (parity, channel) at a swizzled place
    uint16_t* places = reinterpret_cast<uint16_t*>(xch + 1024);   // [128] halfword offset in its segment's packs | length << 12
    unsigned over = 0;
#pragma unroll 1
    for (int r = 0; r < S::kGroups; r++) {
        unsigned cum = 0, min01 = 0, min23 = 0, len01 = 0, len23 = 0;   // packs of this lane's segment so far (halfwords); its channels' header fields
#pragma unroll 1
        for (int rr = 0; rr < S::kPacks / 2; rr++) {
            PackCodes p;
            unsigned lens4;
            int len[4];
            uint64_t wd[4];
            const int q = 2 * rr + par;
            quantise_pack<T, CB, MODE>(lsrc, row_bytes, prm, ord, 64 * r + 16 * q, p);
            over |= p.largest;
            pack_words<BITS>(p, p.mn01, p.mx01, p.mn23, p.mx23, len, lens4, wd);
            constexpr unsigned kMask = ((1u << BITS) - 1u) * 0x00010001u;
            const unsigned l01 = (unsigned)len[0] | ((unsigned)len[1] << 16), l23 = (unsigned)len[2] | ((unsigned)len[3] << 16);
            min01 |= (p.mn01 & kMask) << (q * BITS); min23 |= (p.mn23 & kMask) << (q * BITS);
            len01 |= l01 << (q * LB); len23 |= l23 << (q * LB);
            // packs of the segment and q before this lane's: the other eight lanes', and all of q - 1's for the odd q
            const unsigned sum = (lens4 * 0x01010101u) >> 24;
            unsigned inc = sum;
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) {
                const unsigned n = __shfl_up_sync(0xffffffffu, inc, d, 8);
                if ((lane & 7) >= d) inc += n;
            }
            const unsigned tot = __shfl_sync(0xffffffffu, inc, lane | 7), other = __shfl_xor_sync(0xffffffffu, tot, 16);
            const unsigned at0 = cum + (par ? other : 0u) + inc - sum;
            const unsigned p01 = at0 * 0x00010001u + ((unsigned)len[0] << 16) + (l01 << 12);
            const unsigned p23 = (at0 + len[0] + len[1]) * 0x00010001u + ((unsigned)len[2] << 16) + (l23 << 12);
            cum += tot + other;
            __syncwarp();                                          // the round before has read its words
#pragma unroll
            for (int j = 0; j < 4; j++) words[4 * lane + ((j + (lane >> 2)) & 3)] = make_uint2((unsigned)wd[j], (unsigned)(wd[j] >> 32));
            reinterpret_cast<uint2*>(places)[lane] = make_uint2(p01, p23);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; i++) {                          // the 32 channels of segment i & 1, pack 2 rr + (i >> 1)
                const unsigned place = places[32 * i + lane];
                const uint2 v = words[32 * i + (lane & ~3) + (((lane & 3) + 2 * i + (lane >> 4)) & 3)];
                sts_pack(stage_a + ((i & 1) * S::kGroups + r) * S::kBound + S::kMin + S::kLen + 2 * (place & 0xFFFu), (uint64_t)v.y << 32 | v.x, (int)(place >> 12));
            }
        }
        // the even packs' fields and the odd ones' belong together; half of the lanes store minima, half lengths
        const unsigned m01 = min01 | __shfl_xor_sync(0xffffffffu, min01, 16), m23 = min23 | __shfl_xor_sync(0xffffffffu, min23, 16);
        const unsigned n01 = len01 | __shfl_xor_sync(0xffffffffu, len01, 16), n23 = len23 | __shfl_xor_sync(0xffffffffu, len23, 16);
        uint8_t* seg = stage + (w * S::kGroups + r) * S::kBound;
        if (par == 0) put_fields<S::kPacks * BITS>(seg + (cg & 7) * (S::kPacks * BITS / 2), m01, m23);
        else put_fields<S::kPacks * LB>(seg + S::kMin + (cg & 7) * (S::kPacks * LB / 2), n01, n23);
        if ((lane & 23) == 0) sizes[w * S::kGroups + r] = S::kMin + S::kLen + 2 * cum;
    }
    __syncwarp();
    return over;
}

// Source row (inside a block of CB tokens) of every stored row: the identity, or the caller's reorder of every
// order_block tokens.  NW warps; ends with a CTA barrier.
template <int CB, int NW = 8>
__device__ __forceinline__ void load_row_order(const FusedArgs& a, uint8_t* ord, int b, int cbi) {
    for (int t = threadIdx.x; t < CB; t += 32 * NW) {
        unsigned src = t;
        if (a.order) {
            const int ob = a.order_block, sub = t / ob;
            src = sub * ob + a.order[((int64_t)b * (a.tokens / ob) + (int64_t)cbi * (CB / ob) + sub) * ob + (t - sub * ob)];
        }
        ord[t] = (uint8_t)src;
    }
    __syncthreads();
}

// Form of a V launch: the warps of a CTA, how many CTAs an SM's registers hold, and which way a block takes.  Up to one CTA to an SM: 16 warps with all
// registers.  Up to two: 16 warps twice, through the tile (from registers such a CTA spills).  Beyond: 8 warps, three to an SM (waves of 444 CTAs), or from
// registers four with 64 of them and some spills (waves of 592), where that saves a wave or a CTA has little work.  Of few heads a warp has one block, of
// which the tile is done sooner; where warps are plenty the instructions count, of which registers need fewer.
// us, by CTAs of 148, 296, 444, 592, 600, 888, 1036, 1332, 2048 (fp16; r registers, t tile, warps x CTAs to an SM; - not the form of anything near):
//   4 heads x 64 tokens, 4 bits:  t16x1 17.7 28.7 39.6 46.0 46.2 64.7 74.9 94.9 143   t16x2 17.8 21.8 31.3 32.1 33.1 45.5 54.3 66.4 96.6
//                                 t8x3 19.6 23.2 26.4 36.2 36.3 41.4 53.4 59.4 91.1   r8x3 20.0 24.6 27.9 38.3 38.4 44.1 55.7 62.0 93.9
//                                 r8x4 20.8 25.6 29.6 27.6 34.8 47.1 49.9 65.8 89.9   (900: t8x3 44.2, r8x4 47.4)
//   8 x 64, 4 bits:  t16x1 22.0 35.5 49.6 59.8 60.8 84.2 - 121 183   t16x2 22.1 30.1 48.0 50.2 53.2 71.9 - 103 149   t8x3 24.8 31.6 39.8 62.9 63.2 71.5 - 102 148
//                    r8x3 25.2 31.2 37.9 58.1 58.4 65.5 - 92.7 139   r8x4 28.8 34.6 40.4 46.8 60.4 81.3 - 114 156   (660: t16x2 58.7, r8x3 60.0; 740: 65.8, 62.2)
//   8 x 64, 2 bits (a block's packs are fewer stores; 3 bits alike):  t16x2 27.5 at 296, 45.4 at 600, 55.5 at 740, 126 at 2048; r8x3 29.7, 54.7, 57.6, 131
//   8 x 32:  r16x1 17.0 26.9 36.3 41.7 - 57.5 66.5 - 126   t16x2 17.1 21.3 30.7 32.4 - 44.9 53.5 - 93.7   r8x3 18.5 22.7 26.0 33.9 - 38.1 49.5 - 82.7
//            r8x4 18.3 22.8 26.5 25.7 - 42.1 44.1 - 77.2;  16 x 32: r8x3 23.7 32.3 44.6 62.4 - 81.7 95.7 - 173, t16x2 20.7 31.1 44.6 56.2 - 80.0 92.2 - 171
//   4 x 128: r16x1 24.2 41.1 59.0 73.4 - 105 120 - 227   t8x3 28.4 33.1 55.7 58.3 - 85.2 106 - 184 (of a tile of 128 tokens an SM holds two CTAs)
//            r8x3 29.8 35.5 41.8 68.2 - 75.0 100 - 166   r8x4 33.3 38.1 43.7 52.6 - 93.5 97.0 - 180;  2 x 128 at 2048: r8x3 127, r8x4 125
//   8 x 128: r16x1 30.6 54.8 78.1 97.0 at 592, 304 at 2048; r8x3 39.7 53.1 93.3 97.5, 322; t8x3 37.3 69.3 96.4 128, 414
// Above 8 heads blocks go through the scratch, whole from the tile with aligned stores:
//   16 x 64, 4 bits: t16x1 27.2 at 100, r16x1 27.8; t16x2 54.5 at 296, 102 at 592, 146 at 888, 317 at 2048; t8x3 56.9, 104, 147, 311; r8x3 58.6, 113, 150, 317
//   16 x 64, 2 bits: t16x2 45.1, 80.1, 113, 241; t8x3 49.5, 91.0, 125, 264; r8x3 51.1, 96.5, 127, 268
//   12 x 128, 2 bits: t8x3 73.4, 137 at 592, 436 at 2048, r16x1 73.4, 141, 467 (r8x3 97 at 400, t8x3 110);  16 x 128, 4 bits: r16x1 100, 197, 430 at 1332; t8x3 110, 209, 447
struct VForm { int warps, per_sm; bool tile; };
static VForm v_form(int64_t ctas, int heads, int bits, int cb) {
    const VForm regs3{8, 3, false}, regs4{8, 4, false}, regs_wide{16, 1, false}, tile3{8, 3, true}, tile_two{16, 2, true}, tile_wide{16, 1, true};
    constexpr int64_t n = kSmCount;
    if (ctas <= n) return cb == 64 ? tile_wide : regs_wide;
    const bool one_of_four = ctas > 3 * n && ctas <= 4 * n;           // one wave of four to an SM, two of three
    const bool two_of_four = 4 * ctas > 25 * n && ctas <= 8 * n;      // two, and three of which the last is not near empty
    if (cb == 32) {
        if (heads > 12 || ctas <= 2 * n) return tile_two;
        return one_of_four || (heads <= 8 && ctas > 6 * n) ? regs4 : regs3;
    }
    if (cb == 128) {
        if (heads > 4) return heads <= 8 || heads >= 16 ? regs_wide : ctas > 2 * n && ctas <= 3 * n ? regs3 : tile3;
        if (ctas <= 2 * n) return tile3;
        return one_of_four || two_of_four || (heads <= 2 && ctas > 9 * n) ? regs4 : regs3;
    }
    if (ctas <= 2 * n) return tile_two;
    if (heads > 8) return bits < 4 || one_of_four ? tile_two : tile3;
    if (one_of_four) return regs4;
    if (heads <= 4) return two_of_four || ctas > 9 * n ? regs4 : tile3;
    // (of fewer bits, where the last wave of 444 is up to two of its CTAs to an SM)
    return ctas > 3 * n && (bits < 4 ? (ctas - 1) % (3 * n) < 2 * n : 2 * ctas <= 9 * n) ? tile_two : regs3;
}

// finished blocks that a warp of the V kernel holds in the direct form until their offsets are known
__host__ __device__ constexpr int v_slots(int heads, int nw) { return (2 * heads + nw - 1) / nw; }

constexpr int kVExchange = 1280;   // bytes of a warp's exchange area (see v_block_segments)
// Shared memory of a warp: its tile or exchange area, and `slots` finished blocks, whole or in segments.
template <int CB, int BITS, bool TILE> struct VWarp {
    using S = VSegment<CB, BITS>;
    static constexpr int kWork = TILE ? CB * 64 : kVExchange, kBlock = TILE ? (S::kCount * (2 + S::kBytes) + 15) & ~15 : S::kCount * S::kBound;
    static __host__ __device__ constexpr int bytes(int slots) { return kWork + slots * kBlock; }
};

// NW warps, PER_SM CTAs to an SM, through a tile or from registers: see v_form.  Bound by instructions and the latency of its loads and of the look-back
// (134 M elements, 8 heads x 64 tokens, 4 bits: 130 us from registers, 16.6 instructions per element at 57 % of the issue slots; 138 us through the tile).
// Per 16 tokens x 4 channels of a lane, from registers: quantiser about 300 instructions, pack words 150, exchange, offsets and stores 200.
template <typename T, int BITS, int CB, int NW, int PER_SM, bool TILE>
__global__ void __launch_bounds__(NW * 32, PER_SM) v_fused_encode_kernel(FusedArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = lane_id(), wic = threadIdx.x >> 5;
    const int nctx = a.tokens / CB;
    __shared__ unsigned sh_word, sh_sizes[64];   // bytes of the blocks (TILE), or of the segments of all blocks, in the slots form of a warp's own
    const bool direct = a.status != nullptr;                 // then a warp keeps all of its blocks until the offsets are known
    int cbi = blockIdx.x, b = blockIdx.y;
    if (direct) chain_place(a, &sh_word, b, cbi);
    using S = VSegment<CB, BITS>;
    using W = VWarp<CB, BITS, TILE>;
    const int wstride = W::bytes(direct ? v_slots(a.heads, NW) : 1);
    float4* prm = reinterpret_cast<float4*>(smem);           // [cb] (scale, zero, 1/scale, fast)
    uint8_t* wbase = smem + 32 * CB + wic * wstride;
    const T* xb = reinterpret_cast<const T*>(a.x) + (int64_t)b * a.sb + (int64_t)cbi * CB * a.ss;
    uint8_t* ord = smem + 32 * CB + NW * wstride;
    load_row_order<CB, NW>(a, ord, b, cbi);

    // pass 1: per-token statistics across every head and channel
    constexpr bool kFours = TILE || CB != 64 || PER_SM != 3;   // (v_form: that form is for 5 to 8 heads)
    const TokenState mine = token_params_pass<T, CB, true, NW, kFours>(a, xb, prm, ord, b, cbi, lane, wic);
    // one decision for the whole CTA: the faster conversions need every token's parameters in range
    const bool all_packed = __syncthreads_and(mine.packed);
    const bool all_half = __syncthreads_and(mine.half);

    // pass 2: quantise + pack, one warp per V block
    unsigned seen = 0;
    const int nvb = 2 * a.heads;
    for (int vb = wic; vb < nvb; vb += NW) {
        const T* src = xb + (int64_t)(vb >> 1) * a.sh + 64 * (vb & 1);
        uint8_t* stage = wbase + W::kWork + (direct ? (vb / NW) * W::kBlock : 0);
        const auto slot = [&]() { return a.slots + (((int64_t)b * nctx + cbi) * nvb + vb) * a.slot_stride; };
        const auto put_size = [&](unsigned bytes) { a.info[((int64_t)b * a.info_seq_stride + (int64_t)(a.first_cb + cbi) * nvb + vb) * 2 + 1] = bytes; };
        __syncwarp();
        if constexpr (TILE) {
            seen |= all_half ? v_quantise_tile<T, CB, 2>(src, a.ss, prm, ord, wbase, lane)
                             : all_packed ? v_quantise_tile<T, CB, 1>(src, a.ss, prm, ord, wbase, lane) : v_quantise_tile<T, CB, 0>(src, a.ss, prm, ord, wbase, lane);
            __syncwarp();
            int pos = 2 * S::kCount;                         // behind the table of segment ends
            for (int i = 0; i < S::kCount; i++) {
                const int ch = 32 * (i / S::kGroups) + lane;
                pos += v_pack_segment<CB, BITS>(wbase + ch * CB, v_swz<CB>(ch), i % S::kGroups, stage + pos, lane);
                if (lane == 0) *reinterpret_cast<uint16_t*>(stage + 2 * i) = (uint16_t)(pos - 2 * S::kCount);
            }
            __syncwarp();
            if (direct) {
                if (lane == 0) sh_sizes[vb] = (unsigned)pos;
            } else {
                store_slot(slot(), stage, pos, lane);
                if (lane == 0) put_size((unsigned)pos);
            }
        } else {
            unsigned* sizes = sh_sizes + (direct ? vb : wic) * S::kCount;
            seen |= all_half ? v_block_segments<T, CB, BITS, 2>(src, 2 * (uint64_t)a.ss, prm, ord, stage, wbase, sizes, lane)
                             : all_packed ? v_block_segments<T, CB, BITS, 1>(src, 2 * (uint64_t)a.ss, prm, ord, stage, wbase, sizes, lane)
                                          : v_block_segments<T, CB, BITS, 0>(src, 2 * (uint64_t)a.ss, prm, ord, stage, wbase, sizes, lane);
            if (!direct) {
                store_parts<S::kCount>(slot(), sizes, lane, [&](int i) { return stage + i * S::kBound; });
                if (lane == 0) put_size(parts_size<S::kCount>(sizes));
            }
        }
    }
    if (direct) {
        const auto block = [&](int j) { return smem + 32 * CB + (j % NW) * wstride + W::kWork + (j / NW) * W::kBlock; };
        const int64_t first = (int64_t)(a.first_cb + cbi) * nvb;
        if constexpr (TILE) chain_store(a, b, cbi, sh_sizes, nvb, &sh_word, first, NW, block);
        else chain_store_parts<S::kCount>(a, b, cbi, sh_sizes, nvb, &sh_word, first, NW, [&](int j, int i) { return block(j) + i * S::kBound; });
    }
    const bool bad = mine.bad || (seen & ~(((1u << BITS) - 1u) * 0x00010001u)) != 0;
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags, kFlagCodeRange);
}

// ------------------------------------------------------------------------- K, token mode
// K with per-token parameters (the reference's QuantMethod.PackKV pairing): the parameter pass and
// the quantiser are V's; each warp packs one K block (CB tokens x 128 channels of one
// head) in the K layout, lane = channels 4*lane..4*lane+3, one round per 16 tokens.
template <typename T, int BITS, int CB>
__global__ void __launch_bounds__(256, 3) kt_fused_encode_kernel(FusedArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = lane_id(), wic = threadIdx.x >> 5;
    const int nctx = a.tokens / CB;
    __shared__ unsigned sh_word, sh_sizes[8];
    const bool direct = a.status != nullptr;
    int cbi = blockIdx.x, b = blockIdx.y;
    if (direct) chain_place(a, &sh_word, b, cbi);
    const KGeom g(CB, BITS);
    const int bound16 = (g.head_bytes + g.rounds * (g.min_bytes + g.len_bytes + 128 * 2 * BITS) + 15) & ~15;
    float4* prm = reinterpret_cast<float4*>(smem);
    uint8_t* stage = smem + 32 * CB + wic * bound16;
    const T* xb = reinterpret_cast<const T*>(a.x) + (int64_t)b * a.sb + (int64_t)cbi * CB * a.ss;
    uint8_t* ord = smem + 32 * CB + 8 * bound16;
    load_row_order<CB>(a, ord, b, cbi);

    const TokenState mine = token_params_pass<T, CB>(a, xb, prm, ord, b, cbi, lane, wic);
    // one decision for the whole CTA: the faster conversions need every token's parameters in range
    const bool all_packed = __syncthreads_and(mine.packed);
    const bool all_half = __syncthreads_and(mine.half);

    unsigned seen = 0;
    for (int h = wic; h < a.heads; h += 8) {
        const T* src = xb + (int64_t)h * a.sh + 4 * lane;
        __syncwarp();
        const unsigned stage_a = smem_addr(stage);
        int pos = g.head_bytes;
        const auto rounds = [&](auto mode) {
#pragma unroll 1
            for (int r = 0; r < g.rounds; r++) {
                PackCodes p;
                quantise_pack<T, CB, decltype(mode)::value>(reinterpret_cast<const uint8_t*>(src), 2 * (uint64_t)a.ss, prm, ord, 16 * r, p);
                seen |= p.largest;
                pos += k_pack_round<BITS>(p, p.mn01, p.mn23, p.mn01, p.mx01, p.mn23, p.mx23, stage_a + pos, lane);
                if (lane == 0) *reinterpret_cast<uint16_t*>(stage + 2 * r) = (uint16_t)(pos - g.head_bytes);
            }
        };
        if (all_half) rounds(std::integral_constant<int, 2>{});
        else if (all_packed) rounds(std::integral_constant<int, 1>{});
        else rounds(std::integral_constant<int, 0>{});
        __syncwarp();
        if (direct) {
            if (lane == 0) sh_sizes[h] = (unsigned)pos;     // direct form: at most 8 heads, one block per warp
        } else {
            const int64_t blk = ((int64_t)b * nctx + cbi) * a.heads + h;
            store_slot(a.slots + blk * a.slot_stride, stage, pos, lane);
            if (lane == 0) a.info[((int64_t)b * a.info_seq_stride + (int64_t)(a.first_cb + cbi) * a.heads + h) * 2 + 1] = (unsigned)pos;
        }
    }
    if (direct)
        chain_store(a, b, cbi, sh_sizes, a.heads, &sh_word, (int64_t)(a.first_cb + cbi) * a.heads, 8,
                    [&](int j) { return smem + 32 * CB + j * bound16; });
    const bool bad = mine.bad || (seen & ~(((1u << BITS) - 1u) * 0x00010001u)) != 0;
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags, kFlagCodeRange);
}

// ------------------------------------------------------------------- one block of every sequence
// Launches of one token block per sequence (what leaves the residual in a decode step): their time is the latency of one CTA's
// chain of loads, quantising, packing and storing, so the block is spread over a cluster of `heads` CTAs of four warps, one head
// to a CTA.  A warp holds its rows in registers from one round of loads, packs a round (K) or segments (V) of its own into shared
// memory, and stores it where the sizes of the parts before it put it: inside the CTA through shared memory, across the heads
// through distributed shared memory (no look-back, no scratch).  16 sequences x 64 tokens x 8 heads, four layers' K and V: 98 us
// with one CTA per sequence, 49 us this way.
constexpr int kOneWarps = 4;

// Most CTAs of a one-block launch (us of the general form, then of this one, as both are now).  Blocks of 64 and 128 tokens: up to four to an SM this form is
// ahead, or level (V, 4 heads x 64, 592 CTAs 9.3 and 9.9, 516 8.9 and 7.6); beyond it is ahead still (740 CTAs, 8 heads x 64: K 11.2 and 8.9, V 12.3 and 10.7,
// K with parameters per token 13.8 and 10.7; x 128: K 19.1 and 15.4, V 19.8 and 17.2), but the line was not moved.  Blocks of 32 tokens are
// little work: the form loses once its clusters do not all fit at once, which depends on what a CTA holds and on how many make a cluster, unless the other's one
// CTA per sequence needs a second wave by then.  Where the general form has become faster since the lines were drawn it is up to 12 % ahead below them
// (V, 2 heads: 148 CTAs 4.5 and 4.9; 3 heads: 591 7.2 and 7.6; K with parameters per token, 592: 3 heads 6.3 and 7.1, 8 heads 6.5 and 7.2), level elsewhere.
static int one_block_ctas(int heads, int cb, bool is_v, bool per_token) {
    if (cb != 32 || heads == 1) return 4 * kSmCount;
    if (per_token) return heads <= 3 || (!is_v && heads > 4) ? 4 * kSmCount : 7 * kSmCount / 2;
    return heads == 2 ? 7 * kSmCount / 2 : 3 * kSmCount;
}

// Launched under programmatic stream serialisation: its CTAs are placed while the launch before drains, and touch nothing before
// that one is complete; the launch after it may be placed from here on.
__device__ __forceinline__ void one_block_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The CTA's `n` parts (sizes[], packed at part(i)) of `blocks` equal blocks, n / blocks parts each: tables of part ends, table
// entries and bytes to the stream.  All threads call; two cluster barriers.  `total`: shared word that the other CTAs read.
template <typename Part>
__device__ __forceinline__ void one_block_store(const FusedArgs& a, int b, int blocks, const unsigned* sizes, int n, unsigned* total, int64_t info_first, Part part) {
    cg::cluster_group cluster = cg::this_cluster();
    const int lane = lane_id(), wic = threadIdx.x >> 5, rank = (int)cluster.block_rank(), per = n / blocks, head = 2 * per;
    const unsigned base = a.first_cb == 0 ? 0u : a.stream_bytes[b];    // read by all before the last CTA writes it
    __syncthreads();                                                   // the parts and their sizes are there
    if (threadIdx.x == 0) {
        unsigned sum = (unsigned)(blocks * head);
        for (int i = 0; i < n; i++) sum += sizes[i];
        *total = sum;
    }
    cluster.sync();
    const unsigned other = lane < (int)cluster.num_blocks() ? *cluster.map_shared_rank(total, lane) : 0u;
    const unsigned first = base + warp_sum(lane < rank ? other : 0u), all = base + warp_sum(other);
    if (rank == (int)cluster.num_blocks() - 1 && threadIdx.x == 0) a.stream_bytes[b] = all;
    unsigned off = first;
    for (int blk = 0; blk < blocks; blk++) {
        unsigned size = (unsigned)head;
        for (int i = 0; i < per; i++) size += sizes[blk * per + i];
        if (wic == 0 && lane == 0) {
            uint32_t* bi = a.info + ((int64_t)b * a.info_seq_stride + info_first + blk) * 2;
            bi[0] = off; bi[1] = size;
        }
        if ((int64_t)off + size > a.capacity) {
            if (wic == 0 && lane == 0) atomicOr(a.flags, kFlagStreamOverflow);
        } else {
            uint8_t* dst = a.stream + (int64_t)b * a.stream_seq_stride + off;
            unsigned end = 0;
            for (int i = 0; i < per; i++) {
                const unsigned bytes = sizes[blk * per + i];
                if ((blk * per + i) % kOneWarps == wic) {
                    store_block(dst + head + end, part(blk * per + i), (int)bytes, lane);
                    if (lane == 0) *reinterpret_cast<uint16_t*>(dst + 2 * i) = (uint16_t)(end + bytes);
                }
                end += bytes;
            }
        }
        off += size;
    }
    cluster.sync();                                                    // the others have read `total`
}

// K with per-channel parameters, CB / 16 rounds of 16 tokens dealt to the warps
template <typename T, int BITS, int CB>
__global__ void __launch_bounds__(kOneWarps * 32) k_one_block_kernel(FusedArgs a) {
    one_block_begin();
    constexpr int kRounds = CB / 16, kMine = (kRounds + kOneWarps - 1) / kOneWarps, kBound = (16 * BITS + 16 * len_field_bits(BITS) + 256 * BITS + 15) & ~15;
    using T2 = typename QT<T>::T2;
    __shared__ __align__(16) uint8_t stage[kRounds][kBound];
    __shared__ uint4 extremes[kOneWarps][kLanes];
    __shared__ unsigned sizes[kRounds], total;
    const int lane = lane_id(), wic = threadIdx.x >> 5, h = blockIdx.x, b = blockIdx.y;
    const T* x = reinterpret_cast<const T*>(a.x) + (int64_t)b * a.sb + (int64_t)h * a.sh + 4 * lane;
    uint2 rows[kMine][16];
    T2 lo01 = QT<T>::init2(INFINITY), lo23 = lo01, hi01 = QT<T>::init2(-INFINITY), hi23 = hi01;
#pragma unroll
    for (int i = 0; i < kMine; i++) {
        const int r = wic + kOneWarps * i;
        if (r < kRounds) {
#pragma unroll
            for (int t = 0; t < 16; t++) {
                const int row = a.order ? a.order[(int64_t)b * CB + 16 * r + t] : 16 * r + t;
                rows[i][t] = *reinterpret_cast<const uint2*>(x + (int64_t)row * a.ss);
            }
#pragma unroll
            for (int t = 0; t < 16; t++) {
                const T2 v01 = *reinterpret_cast<const T2*>(&rows[i][t].x), v23 = *reinterpret_cast<const T2*>(&rows[i][t].y);
                lo01 = QT<T>::min2(lo01, v01); hi01 = QT<T>::max2(hi01, v01);
                lo23 = QT<T>::min2(lo23, v23); hi23 = QT<T>::max2(hi23, v23);
            }
        }
    }
    extremes[wic][lane] = make_uint4(*reinterpret_cast<unsigned*>(&lo01), *reinterpret_cast<unsigned*>(&lo23), *reinterpret_cast<unsigned*>(&hi01),
                                     *reinterpret_cast<unsigned*>(&hi23));
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kOneWarps; w++) {
        const uint4 e = extremes[w][lane];
        lo01 = QT<T>::min2(lo01, *reinterpret_cast<const T2*>(&e.x)); lo23 = QT<T>::min2(lo23, *reinterpret_cast<const T2*>(&e.y));
        hi01 = QT<T>::max2(hi01, *reinterpret_cast<const T2*>(&e.z)); hi23 = QT<T>::max2(hi23, *reinterpret_cast<const T2*>(&e.w));
    }
    const Quantiser<T, false> q0(QT<T>::lo_f(lo01), QT<T>::lo_f(hi01), a.rel), q1(QT<T>::hi_f(lo01), QT<T>::hi_f(hi01), a.rel);
    const Quantiser<T, false> q2(QT<T>::lo_f(lo23), QT<T>::lo_f(hi23), a.rel), q3(QT<T>::hi_f(lo23), QT<T>::hi_f(hi23), a.rel);
    if (wic == 0) {
        const int64_t pi = (((int64_t)b * a.heads + h) * a.param_blocks + a.first_block) * 128 + 4 * lane;
        T sc[4] = {QT<T>::cvt(q0.scale), QT<T>::cvt(q1.scale), QT<T>::cvt(q2.scale), QT<T>::cvt(q3.scale)};
        T zr[4] = {QT<T>::cvt(q0.zero), QT<T>::cvt(q1.zero), QT<T>::cvt(q2.zero), QT<T>::cvt(q3.zero)};
        *reinterpret_cast<uint2*>(reinterpret_cast<T*>(a.scale) + pi) = *reinterpret_cast<const uint2*>(sc);
        *reinterpret_cast<uint2*>(reinterpret_cast<T*>(a.zero) + pi) = *reinterpret_cast<const uint2*>(zr);
    }
    bool bad = q0.degenerate() || q1.degenerate() || q2.degenerate() || q3.degenerate();
    const bool packable = __all_sync(0xffffffffu, q0.packable() && q1.packable() && q2.packable() && q3.packable());
    const bool half_ok = __all_sync(0xffffffffu, q0.half_domain() && q1.half_domain() && q2.half_domain() && q3.half_domain());
    const PackedQuantisers<T> pq(q0, q1, q2, q3);
#pragma unroll
    for (int i = 0; i < kMine; i++) {
        const int r = wic + kOneWarps * i;
        if (r < kRounds) {
            const auto row = [&](int t) { return rows[i][t]; };
            unsigned over = 0, size;
            if (half_ok || packable) {
                size = half_ok ? k_encode_round_packed<T, BITS, true>(row, q0, q1, q2, q3, pq, smem_addr(stage[r]), lane, over)
                               : k_encode_round_packed<T, BITS, false>(row, q0, q1, q2, q3, pq, smem_addr(stage[r]), lane, over);
                over &= ~(((1u << BITS) - 1u) * 0x00010001u);
            } else {
                size = k_encode_round<T, BITS>(row, q0, q1, q2, q3, stage[r], lane, over);
            }
            bad = bad || over != 0;
            if (lane == 0) sizes[r] = size;
        }
    }
    one_block_store(a, b, 1, sizes, kRounds, &total, (int64_t)a.first_cb * a.heads + h, [&](int i) { return stage[i]; });
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags, kFlagCodeRange);
}

// Per-token parameters: V (two blocks of 64 channels a head), or K in its own layout (IS_K: one block of 128 channels).  The
// parameters span the heads: every CTA gets the other heads' minima and maxima through distributed shared memory.
template <typename T, int BITS, int CB, bool IS_K>
__global__ void __launch_bounds__(kOneWarps * 32) token_one_block_kernel(FusedArgs a) {
    one_block_begin();
    // packs of 16 tokens: two warps to each half of the channels, which take every other half of the packs
    constexpr int kPacks = CB / 16, kMine = kPacks / 2, kSegs = CB == 128 ? 4 : 2, kParts = IS_K ? kPacks : 2 * kSegs;
    constexpr int kBound = (16 * BITS + 16 * len_field_bits(BITS) + 256 * BITS + 15) & ~15;
    using T2 = typename QT<T>::T2;
    __shared__ __align__(16) uint8_t tile[2 * 64 * CB];
    __shared__ float4 prm[2 * CB];
    __shared__ __align__(16) uint8_t stage[kParts][kBound];
    __shared__ unsigned range[2][CB], sizes[kParts], total;        // range: (minimum, -maximum) of a token, by half; then of this head
    cg::cluster_group cluster = cg::this_cluster();
    const int lane = lane_id(), wic = threadIdx.x >> 5, h = blockIdx.x, b = blockIdx.y;
    const int half = wic & 1, p0 = (wic >> 1) * kMine, r0 = lane >> 3;
    const T* src = reinterpret_cast<const T*>(a.x) + (int64_t)b * a.sb + (int64_t)h * a.sh + 64 * half + 8 * (lane & 7);
    uint4 raw[kMine][4];
#pragma unroll
    for (int i = 0; i < kMine; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int t = 16 * (p0 + i) + 4 * k + r0;
            const int row = a.order ? t / a.order_block * a.order_block + a.order[(int64_t)b * CB + t] : t;
            raw[i][k] = *reinterpret_cast<const uint4*>(src + (int64_t)row * a.ss);
        }
    const auto min_of = [](unsigned x, unsigned y) {
        const T2 m = QT<T>::min2(*reinterpret_cast<const T2*>(&x), *reinterpret_cast<const T2*>(&y));
        return *reinterpret_cast<const unsigned*>(&m);
    };
#pragma unroll
    for (int i = 0; i < kMine; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const T2 v0 = *reinterpret_cast<const T2*>(&raw[i][k].x), v1 = *reinterpret_cast<const T2*>(&raw[i][k].y);
            const T2 v2 = *reinterpret_cast<const T2*>(&raw[i][k].z), v3 = *reinterpret_cast<const T2*>(&raw[i][k].w);
            const T2 lo2 = QT<T>::min2(QT<T>::min2(v0, v1), QT<T>::min2(v2, v3)), hi2 = QT<T>::max2(QT<T>::max2(v0, v1), QT<T>::max2(v2, v3));
            const unsigned l = *reinterpret_cast<const unsigned*>(&lo2), u = *reinterpret_cast<const unsigned*>(&hi2) ^ 0x80008000u;   // -max: one minimum serves both
            unsigned m = min_of(__byte_perm(l, u, 0x5410), __byte_perm(l, u, 0x7632));
#pragma unroll
            for (int s = 4; s > 0; s >>= 1) m = min_of(m, __shfl_xor_sync(0xffffffffu, m, s));
            if ((lane & 7) == 0) range[half][16 * (p0 + i) + 4 * k + r0] = m;
        }
    __syncthreads();
    for (int t = threadIdx.x; t < CB; t += kOneWarps * 32) range[0][t] = min_of(range[0][t], range[1][t]);
    cluster.sync();
    bool bad = false;
    for (int t = threadIdx.x; t < CB; t += kOneWarps * 32) {
        // (a minimum of nothing but NaN is infinity, as in token_params_pass)
        const T2 none = QT<T>::init2(INFINITY);
        unsigned m = *reinterpret_cast<const unsigned*>(&none);
        for (int r = 0; r < a.heads; r++) m = min_of(m, cluster.map_shared_rank(&range[0][0], r)[t]);
        const T2 both = *reinterpret_cast<const T2*>(&m);
        const Quantiser<T, false> qz(QT<T>::lo_f(both), -QT<T>::hi_f(both), a.rel);
        bad = bad || qz.degenerate();
        put_token_params<T, CB>(qz, prm, t);
        if (h == 0) {
            const int64_t pi = (int64_t)b * a.param_tokens + a.first_token + t;
            reinterpret_cast<T*>(a.scale)[pi] = QT<T>::cvt(qz.scale);
            reinterpret_cast<T*>(a.zero)[pi] = QT<T>::cvt(qz.zero);
        }
    }
    __syncthreads();
    bool mine_ok = true, mine_half = true;
    for (int t = threadIdx.x; t < CB; t += kOneWarps * 32) {
        mine_ok = mine_ok && __float_as_uint(prm[t].w) != 0u;
        mine_half = mine_half && reinterpret_cast<const uint4*>(prm + CB)[t].w != 0u;
    }
    const bool all_packed = __syncthreads_and(mine_ok);
    const bool all_half = __syncthreads_and(mine_half);
    unsigned seen = 0;
    const TileLane<CB> out(tile + half * 64 * CB, lane);
    const auto quantise = [&](auto mode) {
#pragma unroll
        for (int i = 0; i < kMine; i++) {
            unsigned c[4][4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                v_quantise_row<T, CB, decltype(mode)::value>(raw[i][k], prm, 16 * (p0 + i) + 4 * k + r0, c[k]);
#pragma unroll
                for (int j = 0; j < 4; j++) seen |= c[k][j];
            }
            out.store(p0 + i, c);
        }
    };
    if (all_half) quantise(std::integral_constant<int, 2>{});
    else if (all_packed) quantise(std::integral_constant<int, 1>{});
    else quantise(std::integral_constant<int, 0>{});
    __syncthreads();
    for (int i = wic; i < kParts; i += kOneWarps) {
        unsigned size;
        if (IS_K) {
            size = kt_pack_round<CB, BITS>(tile, i, stage[i], lane);
        } else {
            // segment i % kSegs of block i / kSegs: 32 channels, then the other 32
            constexpr int kHalfSegs = kSegs / 2;
            const int s = i % kSegs, ch = 32 * (s / kHalfSegs) + lane;
            size = v_pack_segment<CB, BITS>(tile + (i / kSegs) * 64 * CB + ch * CB, v_swz<CB>(ch), s % kHalfSegs, stage[i], lane);
        }
        if (lane == 0) sizes[i] = size;
    }
    constexpr int kBlocks = IS_K ? 1 : 2;
    one_block_store(a, b, kBlocks, sizes, kParts, &total, ((int64_t)a.first_cb * a.heads + h) * kBlocks, [&](int i) { return stage[i]; });
    bad = bad || (seen & ~(((1u << BITS) - 1u) * 0x00010001u)) != 0;
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags, kFlagCodeRange);
}

// ------------------------------------------------------------------------- order from values
// Token order of one block of 64 tokens by descending lower median of the V codes (stable on ties), the
// reference's median_repacking key (utils/compute.py:262-270), computed straight from fp16/bf16 V: per-token
// parameters as in the encoder, the token's heads*128 codes in registers (half a warp per token, 8 heads at
// most), then a binary search for the smallest m with count(code <= m) >= ceil(n / 2).  Same keys and the
// same order as median_order_kernel on the code matrix.  grid (tokens / 64, batch), 256 threads.
template <typename T>
__global__ void __launch_bounds__(256) value_median_order_kernel(FusedArgs a, uint8_t* order) {
    constexpr int CB = 64;
    __shared__ float4 prm[2 * CB];
    __shared__ uint8_t ident[CB];
    __shared__ uint8_t key[CB];
    const int lane = lane_id(), wic = threadIdx.x >> 5;
    const int cbi = blockIdx.x, b = blockIdx.y;
    if (threadIdx.x < CB) ident[threadIdx.x] = (uint8_t)threadIdx.x;
    __syncthreads();
    const T* xb = reinterpret_cast<const T*>(a.x) + (int64_t)b * a.sb + (int64_t)cbi * CB * a.ss;
    token_params_pass<T, CB, false>(a, xb, prm, ident, b, cbi, lane, wic);
    __syncthreads();
    const int need = (a.heads * 128 + 1) / 2;
    const int n_slots = 16 * 64;                       // 16 lanes x 16 words x 4 codes per token; missing heads are filled with large codes
    const unsigned half_mask = 0xFFFFu << (lane & 16);
    for (int t = 2 * wic + (lane >> 4); t < CB; t += 16) {
        const float4 pr = prm[t];
        const uint4 ph = reinterpret_cast<const uint4*>(prm + CB)[t];
        const T* xt = xb + (int64_t)t * a.ss + 8 * (lane & 15);
        unsigned cw[16];
        // The token's codes, four per word.  Parameters inside the checked domain of the element-type quotient: two
        // codes per instruction, as in the encoder; otherwise (or if a code does not fit a byte) one by one in fp32.
        bool wide = ph.w == 0u, small = false;         // small: every code of this lane is known to be at most 15
        if (!wide) {
            HalfQuotient<T> hq;
            hq.r = *reinterpret_cast<const typename QT<T>::T2*>(&ph.x);
            hq.nsp = *reinterpret_cast<const typename QT<T>::T2*>(&ph.y);
            hq.rp = *reinterpret_cast<const typename QT<T>::T2*>(&ph.z);
            hq.kab = ph.w;
            hq.magic = QT<T>::dup((float)(QT<T>::kIntBits == 0x6600u ? 1536 : 192));
            hq.pre = QT<T>::dup(QT<T>::kPre);
            unsigned seen = 0;
#pragma unroll
            for (int h = 0; h < 8; h++) {
                cw[2 * h] = 0x7F7F7F7Fu; cw[2 * h + 1] = 0x7F7F7F7Fu;
                if (h < a.heads) {
                    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(xt + (int64_t)h * a.sh));
                    const unsigned c0 = hq.codes(raw.x), c1 = hq.codes(raw.y), c2 = hq.codes(raw.z), c3 = hq.codes(raw.w);
                    seen |= c0 | c1 | c2 | c3;
                    cw[2 * h] = __byte_perm(c0, c1, 0x6420);
                    cw[2 * h + 1] = __byte_perm(c2, c3, 0x6420);
                }
            }
            wide = (seen & 0xFF80FF80u) != 0u;
            small = (seen & 0xFFF0FFF0u) == 0u;
        }
        if (__ballot_sync(0xffffffffu, wide) & half_mask) {          // the 16 lanes of a token decide together
            Quantiser<T, false> qz;
            qz.scale = pr.x; qz.zero = pr.y;
            qz.prepare();
            const int zi = (int)pr.y;
#pragma unroll
            for (int h = 0; h < 8; h++) {
                cw[2 * h] = 0x7F7F7F7Fu; cw[2 * h + 1] = 0x7F7F7F7Fu;       // heads that do not exist count as large codes
                if (h < a.heads) {
                    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(xt + (int64_t)h * a.sh));
                    const unsigned rw[4] = {raw.x, raw.y, raw.z, raw.w};
                    unsigned c[8];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float2 f = QT<T>::to_float2(rw[i]);
                        c[2 * i] = min(qz.fast ? qz.template code_u8<true>(f.x, zi) : qz.template code_u8<false>(f.x, zi), 127u);
                        c[2 * i + 1] = min(qz.fast ? qz.template code_u8<true>(f.y, zi) : qz.template code_u8<false>(f.y, zi), 127u);
                    }
                    cw[2 * h] = c[0] | (c[1] << 8) | (c[2] << 16) | (c[3] << 24);
                    cw[2 * h + 1] = c[4] | (c[5] << 8) | (c[6] << 16) | (c[7] << 24);
                }
            }
        }
        // count(code <= m) over the token = slots - count(code > m); bit 7 of (code + 127 - m) is set iff code > m
        // (codes are at most 127); the flags of 16 words add up in four byte counters
        auto count_le = [&](int m) {
            const unsigned add = 0x01010101u * (unsigned)(127 - m);
            unsigned acc = 0;
#pragma unroll
            for (int i = 0; i < 16; i++) acc += ((cw[i] + add) >> 7) & 0x01010101u;
            unsigned over = (acc * 0x01010101u) >> 24;               // sum of the four byte counters (each at most 16)
#pragma unroll
            for (int s = 8; s > 0; s >>= 1) over += __shfl_xor_sync(0xffffffffu, over, s);
            return n_slots - (int)over;
        };
        int med = 16;                                  // codes above 15 are not expected (bits <= 4)
        // all of the token's codes at most 15: count_le(15) is the number of real codes, which is at least `need`
        // (decided for the warp's two tokens together: count_le shuffles over the whole warp)
        const bool all_small = __ballot_sync(0xffffffffu, !small) == 0u;
        const bool in_range = all_small || count_le(15) >= need;
        {
            // every lane runs every step (the counts shuffle over the whole warp, whose halves hold different tokens)
            int lo = 0, hi = 15;                       // smallest m in [lo, hi] with count_le(m) >= need
#pragma unroll
            for (int step = 0; step < 4; step++) {
                const int mid = (lo + hi) >> 1;
                if (count_le(mid) >= need) hi = mid; else lo = mid + 1;
            }
            if (in_range) med = hi;
        }
        if ((lane & 15) == 0) key[t] = (uint8_t)med;
    }
    __syncthreads();
    const int i = threadIdx.x;
    if (i < CB) {
        const int ki = key[i];
        int rank = 0;
        for (int j = 0; j < CB; j++) {
            const int kj = key[j];
            rank += (kj > ki) || (kj == ki && j < i);
        }
        order[((int64_t)b * (a.tokens / CB) + cbi) * CB + rank] = (uint8_t)i;
    }
}

// ------------------------------------------------------------------------------------ compact
// one warp per block: slot -> final offset in the sequence's stream
__global__ void __launch_bounds__(kWarpsPerCta * 32) compact_kernel(const uint8_t* slots, int slot_stride, uint8_t* stream,
                                                                    int64_t stream_seq_stride, int64_t capacity, const uint32_t* info,
                                                                    int64_t info_seq_stride, int first_blk, int blocks_per_seq, int batch,
                                                                    int slot_smem, unsigned* flags) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = lane_id(), wic = threadIdx.x >> 5;
    const int64_t warp = (int64_t)blockIdx.x * kWarpsPerCta + wic;
    if (warp >= (int64_t)blocks_per_seq * batch) return;
    const int b = (int)(warp / blocks_per_seq), i = (int)(warp % blocks_per_seq);
    const uint32_t* bi = info + ((int64_t)b * info_seq_stride + first_blk + i) * 2;
    const unsigned off = bi[0], size = bi[1];
    if ((int64_t)off + size > capacity) {
        if (lane == 0) atomicOr(flags, kFlagStreamOverflow);
        return;
    }
    uint8_t* dst = stream + (int64_t)b * stream_seq_stride + off;
    const uint8_t* src = slots + warp * slot_stride;          // 16-byte aligned
    // destination 16-byte chunks: chunk c covers block bytes [16c - phase, 16c - phase + 16)
    const int phase = (int)(reinterpret_cast<uintptr_t>(dst) & 15);   // even
    const int head = min((16 - phase) & 15, (int)size);               // bytes before the first aligned chunk
    for (int j = 2 * lane; j < head; j += 64) *reinterpret_cast<uint16_t*>(dst + j) = *reinterpret_cast<const uint16_t*>(src + j);
    const int nfull = ((int)size - head) >> 4;
    const unsigned* s32 = reinterpret_cast<const unsigned*>(src);
    const int sw = head >> 2;                                          // first source word of the body
    const unsigned sh = (unsigned)(head & 3) * 8;                      // 0 or 16: byte offset inside that word
    for (int c = lane; c < nfull; c += 32) {
        const unsigned* p = s32 + sw + 4 * c;                          // aligned 32-bit loads, realigned by funnel shifts
        const unsigned w0 = p[0], w1 = p[1], w2 = p[2], w3 = p[3], w4 = sh ? p[4] : 0u;   // the fifth word is past the slot when sh == 0
        *reinterpret_cast<uint4*>(dst + head + 16 * c) = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh),
                                                                    __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
    }
    for (int j = head + 16 * nfull + 2 * lane; j < (int)size; j += 64)
        *reinterpret_cast<uint16_t*>(dst + j) = *reinterpret_cast<const uint16_t*>(src + j);
}

// --------------------------------------------------------------------------------------- host
template <typename K>
static int opt_in_smem(K kernel, int bytes) {
    if (bytes > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return kCudaError;
    return kOk;
}

bool fused_encode_applicable(const FusedEncodeRequest& r) {
    if (r.high_precision_zero) return false;   // rare mode: served by the two-stage encoder
    if (r.bits < 2 || r.bits > 4) return false;
    if (r.cb != 32 && r.cb != 64 && r.cb != 128) return false;
    if (r.tokens % r.cb) return false;
    if (r.which == 0 && r.mode == 0 && r.qblock != r.cb) return false;       // K, channel mode: parameters per stream block
    if (r.which == 0 && r.mode != 0 && r.mode != 1) return false;
    if (r.which == 1 && r.mode != 1) return false;                           // V: per-token parameters
    if ((reinterpret_cast<uintptr_t>(r.x) & 15) || (r.stride_b & 7) || (r.stride_h & 7) || (r.stride_s & 7)) return false;
    return true;
}

int64_t fused_encode_scratch_bytes(const FusedEncodeRequest& r) {
    const int nblk = (r.tokens / r.cb) * r.heads * (r.which == 0 ? 1 : 2);
    const int bound = r.which == 0 ? KGeom(r.cb, r.bits).head_bytes + (r.cb / 16) * (16 * r.bits + 16 * len_field_bits(r.bits) + 256 * r.bits)
                                   : VGeom(r.cb, r.bits).head_bytes + VGeom(r.cb, r.bits).nseg * (VGeom(r.cb, r.bits).min_bytes + VGeom(r.cb, r.bits).len_bytes + 32 * VGeom(r.cb, r.bits).ppt * 2 * r.bits);
    return (int64_t)r.batch * nblk * ((bound + 15) & ~15);
}

template <typename T, int BITS>
static int launch_fused_t(const FusedEncodeRequest& r, uint8_t* slots, const uint8_t* order, int order_block, cudaStream_t st) {
    FusedArgs a{};
    a.order = order; a.order_block = order_block;
    a.x = r.x; a.sb = r.stride_b; a.sh = r.stride_h; a.ss = r.stride_s;
    a.scale = r.scale; a.zero = r.zero;
    a.param_blocks = r.param_blocks; a.first_block = r.first_token / r.cb;
    a.param_tokens = r.param_tokens; a.first_token = r.first_token;
    a.slots = slots;
    a.info = r.block_info; a.info_seq_stride = r.info_seq_stride; a.first_cb = r.first_token / r.cb;
    a.batch = r.batch; a.heads = r.heads; a.tokens = r.tokens; a.cb = r.cb; a.bits = BITS; a.rel = r.rel; a.flags = r.flags;
    const int nctx = r.tokens / r.cb;
    int bound16, blocks_per_seq;
    // Direct form: the scratch holds only the ticket and the status array of the look-back.  The slots form stays
    // for more than 8 heads (a CTA of the per-token kernels would not hold all blocks of its token block), for short launches of V in
    // 128-token blocks (short_v), for a scratch too small for the status array, and on request
    // (PKV_ENCODE_PATH=slots: measurements, tests).
    static const bool env_slots = [] { const char* v = std::getenv("PKV_ENCODE_PATH"); return v && std::string(v) == "slots"; }();
    const bool per_token_kernel = r.which == 1 || r.mode == 1;
    const bool k_one = !per_token_kernel && nctx * r.heads <= kKWarpsOne;
    // One token block per sequence and few sequences: one head to a CTA of a cluster (see k_one_block_kernel).
    if (!env_slots && nctx == 1 && r.heads <= 8 && (int64_t)r.batch * r.heads <= one_block_ctas(r.heads, r.cb, r.which == 1, per_token_kernel)) {
        a.stream = r.stream; a.stream_seq_stride = r.stream_seq_stride; a.capacity = r.capacity; a.stream_bytes = reinterpret_cast<unsigned*>(r.stream_bytes);
        const auto by_block = [&](auto cb) {
            constexpr int CB = decltype(cb)::value;
            void (*kern)(FusedArgs) = r.which == 1 ? token_one_block_kernel<T, BITS, CB, false>
                                      : r.mode == 1 ? token_one_block_kernel<T, BITS, CB, true> : k_one_block_kernel<T, BITS, CB>;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(r.heads, r.batch, 1);
            cfg.blockDim = dim3(kOneWarps * 32, 1, 1);
            cfg.stream = st;
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = r.heads;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 2;
            if (cudaLaunchKernelEx(&cfg, kern, a) == cudaSuccess) return (int)kOk;
            cudaGetLastError();
            return (int)kCudaError;
        };
        if (r.cb == 32) return by_block(std::integral_constant<int, 32>{});
        if (r.cb == 64) return by_block(std::integral_constant<int, 64>{});
        return by_block(std::integral_constant<int, 128>{});
    }
    const int links = per_token_kernel ? nctx : k_one ? 1 : (nctx * r.heads + kKWarps - 1) / kKWarps;
    const int64_t chain_bytes = 256 + (int64_t)r.batch * links * 8;
    // V in 128-token blocks, half a CTA to an SM up to two, of few long sequences: all CTAs are there at once, and the chain of a sequence's look-backs is the
    // longest part of the launch (us direct and slots, two sequences, 2 bits: 8 heads, 148 CTAs 29.1 26.9, 296 50.8 47.2; 5 heads 25.0 23.0, 44.3 39.3;
    // 2 heads 21.1 19.1, 26.6 24.2; 4 heads, 4 bits, 24.0 23.3, 33.1 32.8, 370 39.9 41.8; 8 heads, 4 bits, 29.9 30.7, 54.7 55.0; 8 heads, 2 bits, 40 CTAs 24.7 23.3,
    // 20 20.4 20.0, 10 18.5 19.6).  By the blocks of a sequence, slots take of direct's time, 128 or 148 CTAs: 1 block 1.29 to 1.77, 2 0.98 to 1.14, 8 0.96 to 1.04,
    // 32 0.93 to 1.01, 64 0.90 to 0.97, 128 0.87 to 0.93.
    const bool short_v = r.which == 1 && r.cb == 128 && nctx >= 64 && (BITS < 4 || r.heads <= 4) && 2 * (int64_t)r.batch * nctx > kSmCount &&
                         (int64_t)r.batch * nctx <= 2 * kSmCount;
    const bool direct = !env_slots && !short_v && (!per_token_kernel || r.heads <= 8) && chain_bytes <= fused_encode_scratch_bytes(r) &&
                        r.stream_bytes != nullptr;
    if (direct) {
        a.ticket = reinterpret_cast<unsigned*>(slots);
        a.status = reinterpret_cast<unsigned long long*>(slots + 256);
        a.links = links;
        a.stream = r.stream; a.stream_seq_stride = r.stream_seq_stride; a.capacity = r.capacity; a.stream_bytes = reinterpret_cast<unsigned*>(r.stream_bytes);
        if (links > 1 && cudaMemsetAsync(slots, 0, (size_t)chain_bytes, st) != cudaSuccess) return kCudaError;
    }
    if (r.which == 0) {
        const KGeom g(r.cb, BITS);
        bound16 = (g.head_bytes + g.rounds * (g.min_bytes + g.len_bytes + 128 * 2 * BITS) + 15) & ~15;
        a.slot_stride = bound16;
        blocks_per_seq = nctx * r.heads;
        const int64_t nwarps = (int64_t)blocks_per_seq * r.batch;
        const int nw = direct && k_one ? kKWarpsOne : kKWarps, smem = nw * bound16 + 16;
        const unsigned grid = direct ? (unsigned)links * r.batch : (unsigned)((nwarps + nw - 1) / nw);
        if (r.mode == 1) {                       // per-token parameters: CTA per (sequence, token block)
            const int smem_t = 32 * r.cb + 8 * bound16 + r.cb + 16;
            auto launch_kt = [&](auto kern) {
                if (opt_in_smem(kern, smem_t)) return (int)kCudaError;
                kern<<<dim3(nctx, r.batch), 256, smem_t, st>>>(a);
                return (int)kOk;
            };
            int rc = kOk;
            if (r.cb == 32) rc = launch_kt(kt_fused_encode_kernel<T, BITS, 32>);
            else if (r.cb == 64) rc = launch_kt(kt_fused_encode_kernel<T, BITS, 64>);
            else rc = launch_kt(kt_fused_encode_kernel<T, BITS, 128>);
            if (rc != kOk) return rc;
        } else {
            auto launch_k = [&](auto kern) {
                if (opt_in_smem(kern, smem)) return (int)kCudaError;
                kern<<<grid, nw * 32, smem, st>>>(a);
                return (int)kOk;
            };
            const bool one = nw == kKWarpsOne;
            const int rc = a.order ? (one ? launch_k(k_fused_encode_kernel<T, false, BITS, true, kKWarpsOne>) : launch_k(k_fused_encode_kernel<T, false, BITS, true, kKWarps>))
                           : r.stride_s == 128 ? (one ? launch_k(k_fused_encode_kernel<T, true, BITS, false, kKWarpsOne>) : launch_k(k_fused_encode_kernel<T, true, BITS, false, kKWarps>))
                                               : (one ? launch_k(k_fused_encode_kernel<T, false, BITS, false, kKWarpsOne>) : launch_k(k_fused_encode_kernel<T, false, BITS, false, kKWarps>));
            if (rc != kOk) return rc;
        }
    } else {
        const VGeom g(r.cb, BITS);
        bound16 = (g.head_bytes + g.nseg * (g.min_bytes + g.len_bytes + 32 * g.ppt * 2 * BITS) + 15) & ~15;
        a.slot_stride = bound16;
        blocks_per_seq = nctx * 2 * r.heads;
        const VForm form = v_form((int64_t)nctx * r.batch, r.heads, BITS, r.cb);
        const auto launch = [&](auto cb, auto warps, auto per_sm, auto tile) {
            constexpr int CB = decltype(cb)::value, NW = decltype(warps)::value;
            const auto kern = v_fused_encode_kernel<T, BITS, CB, NW, decltype(per_sm)::value, decltype(tile)::value>;
            const int smem = 32 * CB + NW * VWarp<CB, BITS, decltype(tile)::value>::bytes(direct ? v_slots(r.heads, NW) : 1) + CB + 16;
            if (opt_in_smem(kern, smem)) return (int)kCudaError;
            kern<<<dim3(nctx, r.batch), NW * 32, smem, st>>>(a);
            return (int)kOk;
        };
        using std::integral_constant;
        constexpr std::true_type tile{};
        constexpr std::false_type regs{};
        constexpr integral_constant<int, 1> one{};
        constexpr integral_constant<int, 2> two{};
        constexpr integral_constant<int, 3> three{};
        constexpr integral_constant<int, 4> four{};
        constexpr integral_constant<int, 8> eight{};
        constexpr integral_constant<int, 16> sixteen{};
        int rc = kOk;
        const auto by_form = [&](auto cb) {                                         // the forms that v_form gives for the block
            constexpr int CB = decltype(cb)::value;
            if (!form.tile && form.warps == 8) return form.per_sm == 3 ? launch(cb, eight, three, regs) : launch(cb, eight, four, regs);
            if constexpr (CB == 64) {
                if (form.warps == 8) return launch(cb, eight, three, tile);
                return form.per_sm == 1 ? launch(cb, sixteen, one, tile) : launch(cb, sixteen, two, tile);
            } else {
                if (!form.tile) return launch(cb, sixteen, one, regs);
                if constexpr (CB == 32) return launch(cb, sixteen, two, tile);
                else return launch(cb, eight, three, tile);
            }
        };
        if (r.cb == 32) rc = by_form(integral_constant<int, 32>{});
        else if (r.cb == 64) rc = by_form(integral_constant<int, 64>{});
        else rc = by_form(integral_constant<int, 128>{});
        if (rc != kOk) return rc;
    }
    if (direct) return cudaGetLastError() == cudaSuccess ? kOk : kCudaError;
    // offsets: reuse the per-sequence scan of the two-pass encoder
    CodecShape sh{r.batch, r.tokens, r.heads * 128, r.cb, r.which == 0 ? 128 : 64, BITS, r.first_token / r.cb};
    CodecBuffers cbuf{nullptr, 0, r.stream, r.stream_seq_stride, r.capacity, r.block_info, r.info_seq_stride, r.stream_bytes, r.flags};
    int rc = launch_scan_sizes(sh, cbuf, st);
    if (rc != kOk) return rc;
    const int slot_smem = 0;
    const int64_t nwarps = (int64_t)blocks_per_seq * r.batch;
    const int per_cb = r.which == 0 ? r.heads : 2 * r.heads;
    compact_kernel<<<(unsigned)((nwarps + kWarpsPerCta - 1) / kWarpsPerCta), kWarpsPerCta * 32, 0, st>>>(
        slots, a.slot_stride, r.stream, r.stream_seq_stride, r.capacity, r.block_info, r.info_seq_stride, (r.first_token / r.cb) * per_cb,
        blocks_per_seq, r.batch, slot_smem, r.flags);
    return cudaGetLastError() == cudaSuccess ? kOk : kCudaError;
}

template <typename T>
static int launch_fused_b(const FusedEncodeRequest& r, uint8_t* slots, const uint8_t* order, int order_block, cudaStream_t st) {
    switch (r.bits) {
        case 2: return launch_fused_t<T, 2>(r, slots, order, order_block, st);
        case 3: return launch_fused_t<T, 3>(r, slots, order, order_block, st);
        case 4: return launch_fused_t<T, 4>(r, slots, order, order_block, st);
    }
    return kUnsupported;
}

int launch_fused_encode(const FusedEncodeRequest& r, uint8_t* slots, const uint8_t* order, int order_block, cudaStream_t st) {
    if (!fused_encode_applicable(r)) return kUnsupported;
    if (order) {
        // a reorder block must be a whole number of 16-token packs, fit a byte index, divide the stream block
        // and, for K with per-channel parameters, be the stream block itself
        if (order_block < 16 || order_block > 128 || order_block % 16 || r.cb % order_block || r.first_token % order_block) return kUnsupported;
        if (r.which == 0 && r.mode == 0 && order_block != r.cb) return kUnsupported;
        if (reinterpret_cast<uintptr_t>(order) & 15) return kBadArgument;
    }
    if ((int64_t)r.batch * r.tokens == 0) return kOk;
    if (!r.x || !r.scale || !r.zero || !r.stream || !r.block_info || !r.stream_bytes || !r.flags || !slots) return kBadArgument;
    if ((reinterpret_cast<uintptr_t>(slots) & 15) || (reinterpret_cast<uintptr_t>(r.stream) & 1) || (r.stream_seq_stride & 1)) return kBadArgument;
    return r.is_bf16 ? launch_fused_b<__nv_bfloat16>(r, slots, order, order_block, st) : launch_fused_b<__half>(r, slots, order, order_block, st);
}

#ifdef PKV_DEBUG_CHAIN
extern "C" int pkv_debug_chain_stats(unsigned long long* out4, int reset) {
    if (cudaMemcpyFromSymbol(out4, g_chain_stats, 32) != cudaSuccess) return -1;
    if (reset) { unsigned long long z[4] = {0, 0, 0, 0}; cudaMemcpyToSymbol(g_chain_stats, z, 32); }
    return 0;
}
#endif

int launch_value_median_order(const FusedEncodeRequest& r, uint8_t* order, int block, cudaStream_t st) {
    if (block != 64 || r.heads < 1 || r.heads > 8 || r.tokens % 64 || r.high_precision_zero) return kUnsupported;
    if (r.batch < 0 || r.tokens < 0) return kBadArgument;
    if ((int64_t)r.batch * r.tokens == 0) return kOk;
    if (!r.x || !order || (reinterpret_cast<uintptr_t>(r.x) & 15) || (r.stride_b & 7) || (r.stride_h & 7) || (r.stride_s & 7)) return kBadArgument;
    FusedArgs a{};
    a.x = r.x; a.sb = r.stride_b; a.sh = r.stride_h; a.ss = r.stride_s;
    a.batch = r.batch; a.heads = r.heads; a.tokens = r.tokens; a.cb = 64; a.rel = r.rel; a.flags = r.flags;
    if (r.is_bf16) value_median_order_kernel<__nv_bfloat16><<<dim3(r.tokens / 64, r.batch), 256, 0, st>>>(a, order);
    else value_median_order_kernel<__half><<<dim3(r.tokens / 64, r.batch), 256, 0, st>>>(a, order);
    return cudaGetLastError() == cudaSuccess ? kOk : kCudaError;
}

}  // namespace pkv
