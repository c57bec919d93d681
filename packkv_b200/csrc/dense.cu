// Dense view of a layer in one pass: packed stream -> codes -> (code + zero) * scale -> K or V rows in place, with the
// uncompressed residual copied behind them.  This is what the cache returns for a prompt, and for every step when it
// works like the reference's (models/cache/packkv_quant.py:45-85 over utils/compute.py:173-178).
//
// Bound: the 2 bytes per element that it writes (the stream is 0.3 .. 0.6 bytes per element).  The codes stay in
// registers, so memory sees the stream once and the result once; as separate steps (unpack to a cleared code matrix,
// dequantise, concatenate) it also saw 2 bytes of codes and 4 bytes of a second copy per element, in eight launches.
//
// Work split: one warp per stream block (K: cb tokens x 128 channels, V: cb x 64), staged in shared memory; 16 rows of
// one (sequence, head) per warp for the residual.  No warp waits for another.
// Rounding: the code pair leaves the unpack step as bias + code, exact in the element type; taking (bias - minimum) off
// is exact too, and each of the two operations that follow is rounded once to the element type, which equals the
// reference's fp32 operation followed by a rounding (24 bits are at least twice the element's 11 or 8 plus two).
#include "common.cuh"
#include "launch.h"
#include "pack_dev.cuh"

namespace pkv {

template <typename T> struct DT;
template <> struct DT<__half> {
    using T2 = __half2;
    static constexpr unsigned kMagic2 = 0x64006400u, kMagicB = 0x64646464u;     // 0x6400 | c == 1024 + c
    static __device__ __forceinline__ T2 dup(float x) { return __float2half2_rn(x); }
};
template <> struct DT<__nv_bfloat16> {
    using T2 = __nv_bfloat162;
    static constexpr unsigned kMagic2 = 0x43004300u, kMagicB = 0x43434343u;     // 0x4300 | c == 128 + c
    static __device__ __forceinline__ T2 dup(float x) { return __float2bfloat162_rn(x); }
};

template <typename T2> __device__ __forceinline__ unsigned bits_of(const T2& v) { return *reinterpret_cast<const unsigned*>(&v); }
template <typename T2> __device__ __forceinline__ T2 pair_of(unsigned v) { return *reinterpret_cast<const T2*>(&v); }

// (bias + code) pair -> dequantised pair; sub = bias - pack minimum
template <typename T2, bool HP>
__device__ __forceinline__ unsigned dequantise(unsigned biased, T2 sub, T2 scale, T2 zero) {
    const T2 code = __hsub2_rn(pair_of<T2>(biased), sub);
    return bits_of(HP ? __hadd2_rn(__hmul2_rn(code, scale), zero) : __hmul2_rn(__hadd2_rn(code, zero), scale));
}

// Eight codes of `len` bits (code 0 in the top bits of x, anything above bit 8 * len) -> r[k] = (bias + code 7-k, bias + code 3-k)
template <unsigned MAGIC>
__device__ __forceinline__ void unpack_eight(unsigned x, unsigned len, unsigned mask2, unsigned (&r)[4]) {
    unsigned y = ((x << (16u - 4u * len)) & 0xFFFF0000u) | (x & 0x0000FFFFu);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        r[k] = (y & mask2) | MAGIC;
        y >>= len;
    }
}

// Header fields of one lane's four packs: pack minima and lengths as bytes, and the byte offset of each pack.
// Lanes with a length that no encoder writes read as width 0 and set bad.
template <int BITS>
struct PackHeads {
    unsigned mins = 0, lens = 0, total = 0, at[4] = {0, 0, 0, 0};     // as they stand: four packs of width 0, all codes 0
    __device__ __forceinline__ void read(const uint8_t* hdr, int lane, int min_bytes, bool& bad) {
        constexpr int LB = len_field_bits(BITS);
        const unsigned minword = load_lane_field(hdr, lane, 4 * BITS), lenword = load_lane_field(hdr + min_bytes, lane, 4 * LB);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            unsigned len = (lenword >> (j * LB)) & ((1u << LB) - 1u);
            if (len > (unsigned)BITS) { len = 0; bad = true; }
            lens |= len << (8 * j);
            mins |= ((minword >> (j * BITS)) & ((1u << BITS) - 1u)) << (8 * j);
        }
        const unsigned inc = warp_inclusive_sum(lens), tot = __shfl_sync(0xffffffffu, inc, 31), exc = inc - lens;
        unsigned before = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            at[j] = 2 * (before + ((exc >> (8 * j)) & 0xFFu));
            before += (tot >> (8 * j)) & 0xFFu;
        }
        total = 2 * before;
    }
};

// the lane's pack j as two groups of eight biased pairs
template <unsigned MAGIC>
__device__ __forceinline__ void unpack_pack(const uint8_t* pack, unsigned len, unsigned (&a)[4], unsigned (&b)[4]) {
    unsigned lo, hi;
    load_u64_smem_align2(pack, lo, hi);
    const unsigned mask2 = ((1u << len) - 1u) * 0x00010001u;
    unpack_eight<MAGIC>(__byte_perm(lo, hi, 0x3210u + 0x1111u * len), len, mask2, a);   // tokens 0..7
    unpack_eight<MAGIC>(lo, len, mask2, b);                                             // tokens 8..15
}

// Per-token parameters of a block in pair order, words [8-token group][k] = (token 7-k, token 3-k)
template <typename T>
__device__ __forceinline__ void load_token_params(const pkv_dense_args& a, int b, int first, int cb, unsigned* scale, unsigned* zero, int lane) {
    const uint16_t* s = reinterpret_cast<const uint16_t*>(a.scale) + (int64_t)b * a.param_tokens + first;
    const uint16_t* z = reinterpret_cast<const uint16_t*>(a.zero) + (int64_t)b * a.param_tokens + first;
    for (int i = lane; i < cb / 2; i += 32) {
        const int t = 8 * (i >> 2) + 3 - (i & 3);
        scale[i] = s[t + 4] | ((unsigned)s[t] << 16);
        zero[i] = z[t + 4] | ((unsigned)z[t] << 16);
    }
}

// Whether a reorder group of n entries names every row of the group once.  Warp-cooperative.
__device__ __forceinline__ bool is_permutation(const uint8_t* group, int n, int lane) {
    bool ok = true;
    for (int w = 0; w < n; w += 32) {                 // rows w .. w + 31
        unsigned seen = 0;
        for (int i = lane; i < n; i += 32) {
            const unsigned v = group[i] - (unsigned)w;
            if (v < 32u) seen |= 1u << v;
        }
        ok = __reduce_or_sync(0xffffffffu, seen) == (n - w >= 32 ? 0xffffffffu : (1u << (n - w)) - 1u) && ok;
    }
    return ok;
}

// Row, relative to the stream block's first, of every token of the block.  The reorder moves tokens inside groups of
// order_block, which may begin or end in another block.  Its entries say where rows are stored, so a group that is no
// permutation (a corrupt blob) stays in stored order: every row is written, none outside its group.  False if there is one.
__device__ __forceinline__ bool place_rows(const pkv_dense_args& a, int b, int cbi, int16_t* place, int lane) {
    const int first = cbi * a.cb, ob = a.order_block;
    for (int t = lane; t < a.cb; t += 32) place[t] = (int16_t)t;
    if (!a.order || ob == 1) return true;
    __syncwarp();
    bool ok = true;
    const uint8_t* ord = a.order + (int64_t)b * a.order_seq_stride;
    for (int g = first / ob * ob; g < first + a.cb; g += ob) {
        if (!is_permutation(ord + g, ob, lane)) { ok = false; continue; }
        for (int i = lane; i < ob; i += 32)
            if (g + i >= first && g + i < first + a.cb) place[g + i - first] = (int16_t)(g - first + ord[g + i]);
    }
    return ok;
}

// 16 residual rows of one (sequence, head) behind the dequantised ones
__device__ __forceinline__ void copy_residual(const pkv_dense_args& a, int64_t item, int lane) {
    const int per = (a.n_res + 15) >> 4, chunks = a.dim >> 3;
    const int row0 = (int)(item % per) * 16, rows = min(16, a.n_res - row0);
    const int64_t bh = item / per;
    const int b = (int)(bh / a.heads), h = (int)(bh % a.heads);
    const uint16_t* src = reinterpret_cast<const uint16_t*>(a.res) + b * a.res_stride_b + h * a.res_stride_h + (int64_t)row0 * 128;
    uint16_t* dst = reinterpret_cast<uint16_t*>(a.out) + b * a.o_stride_b + h * a.o_stride_h + (int64_t)(a.n_comp + row0) * a.o_stride_s;
    for (int i = lane; i < rows * chunks; i += 32) {
        const int r = i / chunks, c = i % chunks;
        *reinterpret_cast<uint4*>(dst + r * a.o_stride_s + 8 * c) = *reinterpret_cast<const uint4*>(src + r * 128 + 8 * c);
    }
}

template <int WHICH>
__host__ __device__ int dense_bound(int cb, int bits) {
    if (WHICH == 0) {
        const KGeom g(cb, bits);
        return g.head_bytes + g.rounds * (g.min_bytes + g.len_bytes + 128 * 2 * bits);
    }
    const VGeom g(cb, bits);
    return g.head_bytes + g.nseg * (g.min_bytes + g.len_bytes + 32 * g.ppt * 2 * bits);
}
// the block, its token parameters, and in the general form the row of every token
template <int WHICH, bool GENERAL>
__host__ __device__ int dense_slot(int cb, int bits) { return ((dense_bound<WHICH>(cb, bits) + 48 + 15) & ~15) + 4 * cb + (GENERAL ? 2 * cb : 0); }

// WHICH 0: K, parameters per (head, block, channel) or, with TOKEN, per token; WHICH 1: V, per token.
// GENERAL: layers that are reordered, or whose channel parameters change inside a stream block or span several.  Rows come
// from a table in shared memory (V of 4 x 8064 tokens x 8 heads, 4 bits: 33 us; 50 with a division and a byte of the order
// for every row); plain layers keep a kernel without either (27 us; 34 with the order as a run-time branch).
template <typename T, int WHICH, int BITS, bool HP, bool TOKEN, bool GENERAL>
__global__ void __launch_bounds__(kWarpsPerCta * 32) dense_kernel(pkv_dense_args a) {
    using T2 = typename DT<T>::T2;
    constexpr unsigned MAGIC = DT<T>::kMagic2;
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = lane_id(), wic = threadIdx.x >> 5;
    const int nblk = WHICH == 0 ? a.heads : 2 * a.heads;
    const int64_t per_seq = (int64_t)(a.n_comp / a.cb) * nblk, blocks = per_seq * a.batch;
    int64_t item = (int64_t)blockIdx.x * kWarpsPerCta + wic;
    if (item >= blocks) {
        item -= blocks;
        if (item < (int64_t)a.batch * a.heads * ((a.n_res + 15) >> 4)) copy_residual(a, item, lane);
        return;
    }
    const int b = (int)(item / per_seq), rem = (int)(item % per_seq), cbi = rem / nblk, hb = rem % nblk;
    const int h = WHICH == 0 ? hb : hb >> 1;
    uint8_t* slot = smem + wic * dense_slot<WHICH, GENERAL>(a.cb, BITS);
    unsigned* tscale = reinterpret_cast<unsigned*>(slot + dense_slot<WHICH, false>(a.cb, BITS) - 4 * a.cb);
    unsigned* tzero = tscale + a.cb / 2;
    int16_t* place = reinterpret_cast<int16_t*>(tzero + a.cb / 2);
    const uint32_t* bi = a.block_info + (b * a.info_seq_stride + rem) * 2;
    const unsigned off = bi[0], size = bi[1];
    if (TOKEN) load_token_params<T>(a, b, cbi * a.cb, a.cb, tscale, tzero, lane);
    T2 cscale[4], czero[4];
    const auto channel_params = [&](int t) {          // of token t of this block
        const int64_t pi = (((int64_t)b * a.heads + h) * a.param_blocks + (GENERAL ? (cbi * a.cb + t) / a.qblock : cbi)) * 128 + 4 * lane;
        const uint2 s = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const T*>(a.scale) + pi));
        const uint2 z = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const T*>(a.zero) + pi));
#pragma unroll
        for (int j = 0; j < 4; j++) {
            cscale[j] = pair_of<T2>(__byte_perm(j < 2 ? s.x : s.y, 0, (j & 1) ? 0x3232 : 0x1010));
            czero[j] = pair_of<T2>(__byte_perm(j < 2 ? z.x : z.y, 0, (j & 1) ? 0x3232 : 0x1010));
        }
    };
    if (!TOKEN) channel_params(0);
    // a block that the table places outside the stream, or that is cut short, reads as codes 0 from there on
    bool bad = (int64_t)off + size > a.capacity || (int)size > dense_bound<WHICH>(a.cb, BITS) || (int)size < (WHICH == 0 ? a.cb / 8 : a.cb == 128 ? 8 : 4);
    const uint8_t* blk = slot;
    if (!bad) {
        const uint8_t* base = a.stream + b * a.stream_seq_stride;
        blk = warp_copy_in(slot, base + off, (int)size, lane, base, base + a.capacity);
    }
    bool cut = bad;
    T* out = reinterpret_cast<T*>(a.out) + b * a.o_stride_b + h * a.o_stride_h + (int64_t)cbi * a.cb * a.o_stride_s;
    if (GENERAL) bad |= !place_rows(a, b, cbi, place, lane);
    __syncwarp();
    const auto row = [&](int t) { return out + (GENERAL ? place[t] : t) * a.o_stride_s; };   // of stored token t of this block
    const T2 bias = DT<T>::dup(MAGIC == 0x64006400u ? 1024.f : 128.f);

    if (WHICH == 0) {
        const KGeom g(a.cb, BITS);
        int pos = g.head_bytes;
        const bool inside = 4 * lane < a.dim;
        for (int r = 0; r < g.rounds; r++) {
            if (GENERAL && !TOKEN && a.qblock != a.cb && r > 0) channel_params(16 * r);
            unsigned u[4][2][4] = {};                     // [channel][group of eight][k]
            if (!cut && pos + g.min_bytes + g.len_bytes <= (int)size) {
                PackHeads<BITS> ph;
                ph.read(blk + pos, lane, g.min_bytes, bad);
                const uint8_t* packs = blk + pos + g.min_bytes + g.len_bytes;
                pos += g.min_bytes + g.len_bytes + ph.total;
                cut = pos > (int)size;
                if (!cut) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        unpack_pack<MAGIC>(packs + ph.at[j], (ph.lens >> (8 * j)) & 0xFFu, u[j][0], u[j][1]);
                        const T2 sub = __hsub2_rn(bias, __hsub2_rn(pair_of<T2>(__byte_perm(ph.mins, DT<T>::kMagicB, 0x4040 + 0x0101 * j)), bias));
#pragma unroll
                        for (int e = 0; e < 2; e++)
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                u[j][e][k] = TOKEN ? dequantise<T2, HP>(u[j][e][k], sub, pair_of<T2>(tscale[8 * r + 4 * e + k]), pair_of<T2>(tzero[8 * r + 4 * e + k]))
                                                   : dequantise<T2, HP>(u[j][e][k], sub, cscale[j], czero[j]);
                    }
                }
            } else {
                cut = true;
            }
            if (cut) {
                bad = true;
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int e = 0; e < 2; e++)
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            u[j][e][k] = TOKEN ? dequantise<T2, HP>(MAGIC, bias, pair_of<T2>(tscale[8 * r + 4 * e + k]), pair_of<T2>(tzero[8 * r + 4 * e + k]))
                                               : dequantise<T2, HP>(MAGIC, bias, cscale[j], czero[j]);
            }
            if (inside) {
#pragma unroll
                for (int e = 0; e < 2; e++)
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int t = 16 * r + 8 * e + 3 - k;
                        *reinterpret_cast<uint2*>(row(t) + 4 * lane) = make_uint2(__byte_perm(u[0][e][k], u[1][e][k], 0x7632), __byte_perm(u[2][e][k], u[3][e][k], 0x7632));
                        *reinterpret_cast<uint2*>(row(t + 4) + 4 * lane) = make_uint2(__byte_perm(u[0][e][k], u[1][e][k], 0x5410), __byte_perm(u[2][e][k], u[3][e][k], 0x5410));
                    }
            }
        }
    } else {
        // a lane holds one channel; neighbours exchange so that the even lane stores both channels of the earlier
        // token of a pair and the odd lane those of the later one
        const VGeom g(a.cb, BITS);
        const int odd = lane & 1;
        int pos = g.head_bytes;
        for (int w = 0; w < 2; w++) {
            const int ch = 64 * (hb & 1) + 32 * w + (lane & ~1);
            const bool inside = ch < a.dim;
            for (int r = 0; r < g.rpw; r++) {
                PackHeads<BITS> ph;
                const uint8_t* packs = slot;
                if (!cut && pos + g.min_bytes + g.len_bytes <= (int)size) {
                    ph.read(blk + pos, lane, g.min_bytes, bad);
                    packs = blk + pos + g.min_bytes + g.len_bytes;
                    pos += g.min_bytes + g.len_bytes + ph.total;
                    cut = pos > (int)size;
                } else {
                    cut = true;
                }
                if (cut) {
                    bad = true;
                    ph = PackHeads<BITS>();
                    packs = slot;
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    unsigned u[2][4];
                    unpack_pack<MAGIC>(packs + ph.at[q], (ph.lens >> (8 * q)) & 0xFFu, u[0], u[1]);
                    const T2 sub = __hsub2_rn(bias, __hsub2_rn(pair_of<T2>(__byte_perm(ph.mins, DT<T>::kMagicB, 0x4040 + 0x0101 * q)), bias));
                    const int t0 = 64 * r + 16 * q;
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const uint4 s4 = *reinterpret_cast<const uint4*>(tscale + t0 / 2 + 4 * e), z4 = *reinterpret_cast<const uint4*>(tzero + t0 / 2 + 4 * e);
                        const unsigned sc[4] = {s4.x, s4.y, s4.z, s4.w}, ze[4] = {z4.x, z4.y, z4.z, z4.w};
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const unsigned mine = dequantise<T2, HP>(u[e][k], sub, pair_of<T2>(sc[k]), pair_of<T2>(ze[k]));
                            const unsigned theirs = __shfl_xor_sync(0xffffffffu, mine, 1);
                            const int t = t0 + 8 * e + 3 - k + 4 * odd;
                            if (inside) *reinterpret_cast<unsigned*>(row(t) + ch) = odd ? __byte_perm(theirs, mine, 0x5410) : __byte_perm(mine, theirs, 0x7632);
                        }
                    }
                }
            }
        }
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.flags, kFlagBadStream);
}

template <typename T, int WHICH, int BITS, bool HP, bool TOKEN, bool GENERAL>
static int start(const pkv_dense_args& a, cudaStream_t st) {
    const auto kern = dense_kernel<T, WHICH, BITS, HP, TOKEN, GENERAL>;
    const int smem = kWarpsPerCta * dense_slot<WHICH, GENERAL>(a.cb, BITS);
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return kCudaError;
    const int64_t items = (int64_t)a.batch * ((int64_t)(a.n_comp / a.cb) * (WHICH == 0 ? a.heads : 2 * a.heads) + (int64_t)a.heads * ((a.n_res + 15) >> 4));
    const int64_t ctas = (items + kWarpsPerCta - 1) / kWarpsPerCta;
    if (ctas > 0x7FFFFFFF) return kBadArgument;
    kern<<<(unsigned)ctas, kWarpsPerCta * 32, smem, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? kOk : kCudaError;
}

template <typename T, int WHICH, int BITS, bool HP, bool TOKEN>
static int pick_form(const pkv_dense_args& a, cudaStream_t st) {
    const bool general = a.order || (!TOKEN && a.qblock != a.cb);
    return general ? start<T, WHICH, BITS, HP, TOKEN, true>(a, st) : start<T, WHICH, BITS, HP, TOKEN, false>(a, st);
}
template <typename T, int WHICH, int BITS, bool TOKEN>
static int pick_zero(const pkv_dense_args& a, cudaStream_t st) {
    return a.high_precision_zero ? pick_form<T, WHICH, BITS, true, TOKEN>(a, st) : pick_form<T, WHICH, BITS, false, TOKEN>(a, st);
}
template <typename T, int BITS>
static int pick_mode(const pkv_dense_args& a, cudaStream_t st) {
    if (a.which == 1) return pick_zero<T, 1, BITS, true>(a, st);
    return a.mode == PKV_K_TOKEN ? pick_zero<T, 0, BITS, true>(a, st) : pick_zero<T, 0, BITS, false>(a, st);
}
template <typename T>
static int pick_bits(const pkv_dense_args& a, cudaStream_t st) {
    return a.bits == 2 ? pick_mode<T, 2>(a, st) : a.bits == 3 ? pick_mode<T, 3>(a, st) : pick_mode<T, 4>(a, st);
}

int launch_dense(const pkv_dense_args& a, cudaStream_t st) {
    if ((a.which != 0 && a.which != 1) || a.batch < 0 || a.heads <= 0 || a.n_comp < 0 || a.n_res < 0 || a.dim <= 0) return kBadArgument;
    if (a.bits < 2 || a.bits > 4 || (a.cb != 64 && a.cb != 128) || (a.mode != PKV_K_CHANNEL && a.mode != PKV_K_TOKEN) || a.dim > 128 || a.dim % 8) return kUnsupported;
    // a round of 16 tokens has one set of channel parameters
    if (a.which == 1 ? a.mode != PKV_K_TOKEN : a.mode == PKV_K_CHANNEL && (a.qblock <= 0 || a.qblock % 16)) return kUnsupported;
    if (a.n_comp % a.cb) return kBadArgument;
    if ((int64_t)a.batch * ((int64_t)a.n_comp + a.n_res) == 0) return kOk;
    // rows are written in 8-byte (K) and 16-byte (residual) pieces
    const auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (!a.out || !a.flags || !aligned(a.out) || ((a.o_stride_b | a.o_stride_h | a.o_stride_s) & 7)) return kBadArgument;
    if (a.n_res && (!a.res || !aligned(a.res) || ((a.res_stride_b | a.res_stride_h) & 7))) return kBadArgument;
    if (a.n_comp) {
        if (!a.stream || !a.block_info || !a.scale || !a.zero || (reinterpret_cast<uintptr_t>(a.stream) & 1) || (a.stream_seq_stride & 1)) return kBadArgument;
        if (a.mode == PKV_K_CHANNEL ? a.n_comp % a.qblock || a.param_blocks < a.n_comp / a.qblock || (reinterpret_cast<uintptr_t>(a.scale) & 7) || (reinterpret_cast<uintptr_t>(a.zero) & 7)
                                    : a.param_tokens < a.n_comp) return kBadArgument;
        if (a.order && (a.order_block <= 0 || a.order_block > 256 || a.n_comp % a.order_block || a.order_seq_stride < a.n_comp)) return kBadArgument;
    }
    return a.is_bf16 ? pick_bits<__nv_bfloat16>(a, st) : pick_bits<__half>(a, st);
}

}  // namespace pkv
