// Small kernels of the cache's append path.
//   rows        : new tokens to where they are kept: K through the rotary embedding, op for op like the reference's
//                 apply_rotary_pos_emb_single (utils/compute.py:22-43): (t*cos) + (rotate_half(t)*sin), each op
//                 rounded to the element type; V copied.  One launch.
//   dequantize  : codes + scale/zero -> dense K or V exactly as the reference's cache does it,
//                 (code + zero) * scale or code * scale + min (utils/compute.py:173-178), for codes of any
//                 quantisation mode; a packed layer goes through dense.cu instead.
#include "common.cuh"
#include "launch.h"

namespace pkv {

template <typename T> struct CT;
template <> struct CT<__half> {
    static __device__ __forceinline__ float ld(const __half* p) { return __half2float(*p); }
    static __device__ __forceinline__ float rnd(float x) { return __half2float(__float2half_rn(x)); }
    static __device__ __forceinline__ __half cvt(float x) { return __float2half_rn(x); }
};
template <> struct CT<__nv_bfloat16> {
    static __device__ __forceinline__ float ld(const __nv_bfloat16* p) { return __bfloat162float(*p); }
    static __device__ __forceinline__ float rnd(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
    static __device__ __forceinline__ __nv_bfloat16 cvt(float x) { return __float2bfloat16_rn(x); }
};

// Rows of new tokens: K rotated (cos != null) or copied, V copied (v != null), from (B, H, T, dim) in any strides to rows of
// `width` channels; channels dim .. width-1 repeat the row's first ones, or are zero.  Used for the rotated prompt, the
// residual's new rows, the widened rows of heads below 128 channels and the padded q of such heads.
// Bound: memory on a prompt (2 bytes read and written per element), launch latency on a decode step.  A thread takes eight
// channels of each half of a row, so that the rotation's partner is its own, in 16-byte accesses, and keeps the cosines for
// `hpt` heads of its token.  One channel to a thread, as before, took 70 us for K of 4 x 8191 tokens x 8 heads (floor 20).
template <typename T>
__device__ __forceinline__ uint4 rotate8(const uint4& x, const uint4& partner, float sign, const uint4& cos, const uint4& sin) {
    const T *xe = reinterpret_cast<const T*>(&x), *pe = reinterpret_cast<const T*>(&partner);
    const T *ce = reinterpret_cast<const T*>(&cos), *se = reinterpret_cast<const T*>(&sin);
    uint4 out;
    T* o = reinterpret_cast<T*>(&out);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float a = CT<T>::rnd(CT<T>::ld(xe + i) * CT<T>::ld(ce + i));
        const float c = CT<T>::rnd(sign * CT<T>::ld(pe + i) * CT<T>::ld(se + i));
        o[i] = CT<T>::cvt(a + c);
    }
    return out;
}

template <typename T>
__global__ void __launch_bounds__(256) rows_kernel(RowsArgs r, int hpt, unsigned items) {
    const unsigned id = blockIdx.x * 256u + threadIdx.x;
    if (id >= items) return;
    const int per_row = r.dim >> 4, groups = (r.heads + hpt - 1) / hpt, half = r.dim >> 1, tail = r.width - r.dim;
    const int c = (int)(id % per_row), hg = (int)(id / per_row % groups), bt = (int)(id / per_row / groups), t = bt % r.tokens, b = bt / r.tokens;
    const int d0 = 8 * c, d1 = half + 8 * c;
    uint4 c0, c1, s0, s1;
    if (r.cos) {
        const int64_t at = b * r.cs_stride_b + (int64_t)t * r.dim;
        const T *cs = reinterpret_cast<const T*>(r.cos) + at, *sn = reinterpret_cast<const T*>(r.sin) + at;
        c0 = __ldg(reinterpret_cast<const uint4*>(cs + d0)); c1 = __ldg(reinterpret_cast<const uint4*>(cs + d1));
        s0 = __ldg(reinterpret_cast<const uint4*>(sn + d0)); s1 = __ldg(reinterpret_cast<const uint4*>(sn + d1));
    }
    const auto put = [&](T* row, const uint4& v0, const uint4& v1) {
        const uint4 zero = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(row + d0) = v0;
        *reinterpret_cast<uint4*>(row + d1) = v1;
        if (d0 < tail) *reinterpret_cast<uint4*>(row + r.dim + d0) = r.zero_tail ? zero : v0;
        if (d1 < tail) *reinterpret_cast<uint4*>(row + r.dim + d1) = r.zero_tail ? zero : v1;
    };
    for (int h = hg * hpt; h < min(r.heads, (hg + 1) * hpt); h++) {
        const T* x = reinterpret_cast<const T*>(r.k) + b * r.k_stride_b + h * r.k_stride_h + t * r.k_stride_s;
        const int64_t o = b * r.o_stride_b + h * r.o_stride_h + (r.position + t) * r.o_stride_s;
        uint4 x0 = *reinterpret_cast<const uint4*>(x + d0), x1 = *reinterpret_cast<const uint4*>(x + d1), y0, y1;
        if (r.v) {
            const T* y = reinterpret_cast<const T*>(r.v) + b * r.v_stride_b + h * r.v_stride_h + t * r.v_stride_s;
            y0 = *reinterpret_cast<const uint4*>(y + d0); y1 = *reinterpret_cast<const uint4*>(y + d1);
        }
        if (r.cos) {
            const uint4 r0 = rotate8<T>(x0, x1, -1.f, c0, s0), r1 = rotate8<T>(x1, x0, 1.f, c1, s1);
            x0 = r0; x1 = r1;
        }
        put(reinterpret_cast<T*>(r.k_out) + o, x0, x1);
        if (r.v) put(reinterpret_cast<T*>(r.v_out) + o, y0, y1);
    }
}

// The same rows one channel at a time, for sizes, strides and addresses that 16-byte accesses do not fit.
// grid (tokens, heads, batch), 128 threads = channels of the written row
template <typename T>
__global__ void __launch_bounds__(128) rows_scalar_kernel(RowsArgs r) {
    const int t = blockIdx.x, h = blockIdx.y, b = blockIdx.z, w = threadIdx.x;
    if (w >= r.width) return;
    const int d = w < r.dim ? w : w - r.dim, half = r.dim / 2;
    const bool zero = r.zero_tail && w >= r.dim;
    const T* x = reinterpret_cast<const T*>(r.k) + b * r.k_stride_b + h * r.k_stride_h + t * r.k_stride_s;
    const int64_t o = b * r.o_stride_b + h * r.o_stride_h + (r.position + t) * r.o_stride_s + w;
    T kv = x[d];
    if (r.cos) {
        const int64_t at = b * r.cs_stride_b + (int64_t)t * r.dim + d;
        const float rot = d < half ? -CT<T>::ld(x + d + half) : CT<T>::ld(x + d - half);
        const float a = CT<T>::rnd(CT<T>::ld(x + d) * CT<T>::ld(reinterpret_cast<const T*>(r.cos) + at));
        const float c = CT<T>::rnd(rot * CT<T>::ld(reinterpret_cast<const T*>(r.sin) + at));
        kv = CT<T>::cvt(a + c);
    }
    reinterpret_cast<T*>(r.k_out)[o] = zero ? CT<T>::cvt(0.f) : kv;
    if (r.v) {
        const T* y = reinterpret_cast<const T*>(r.v) + b * r.v_stride_b + h * r.v_stride_h + t * r.v_stride_s;
        reinterpret_cast<T*>(r.v_out)[o] = zero ? CT<T>::cvt(0.f) : y[d];
    }
}

// grid (tokens, heads, batch), 128 threads = channels
template <typename T, bool HP>
__global__ void __launch_bounds__(128) dequant_kernel(DequantArgs q) {
    const int t = blockIdx.x, h = blockIdx.y, b = blockIdx.z, d = threadIdx.x;
    const float code = (float)q.codes[(int64_t)b * q.codes_seq_stride + (int64_t)t * (q.heads * 128) + h * 128 + d];
    int64_t pi;
    if (q.mode == 0) pi = (((int64_t)b * q.heads + h) * q.param_blocks + (q.first_token + t) / q.block) * 128 + d;
    else if (q.mode == 1) pi = (int64_t)b * q.param_tokens + q.first_token + t;
    else if (q.mode == 2) pi = ((int64_t)b * q.heads + h) * q.param_tokens + q.first_token + t;      // vector: per (head, token)
    else pi = (int64_t)b * q.param_blocks + (q.first_token + t) / q.block;                           // block: per token block
    const float s = CT<T>::ld(reinterpret_cast<const T*>(q.scale) + pi), z = CT<T>::ld(reinterpret_cast<const T*>(q.zero) + pi);
    const float v = HP ? CT<T>::rnd(CT<T>::rnd(code * s) + z) : CT<T>::rnd(CT<T>::rnd(code + z) * s);
    reinterpret_cast<T*>(q.out)[(int64_t)b * q.o_stride_b + (int64_t)h * q.o_stride_h + (int64_t)t * q.o_stride_s + d] = CT<T>::cvt(v);
}

int launch_rows(const RowsArgs& r, cudaStream_t st) {
    if (r.batch < 0 || r.heads <= 0 || r.tokens < 0 || r.position < 0 || r.position + (int64_t)r.tokens > r.capacity) return kBadArgument;
    if (r.dim <= 0 || r.width > 128 || r.width < r.dim || r.width - r.dim > r.dim || (r.cos && (r.dim & 1))) return kBadArgument;
    if ((int64_t)r.batch * r.tokens == 0) return kOk;
    if (!r.k || !r.k_out || ((r.v == nullptr) != (r.v_out == nullptr)) || ((r.cos == nullptr) != (r.sin == nullptr))) return kBadArgument;
    const uintptr_t at = reinterpret_cast<uintptr_t>(r.k) | reinterpret_cast<uintptr_t>(r.v) | reinterpret_cast<uintptr_t>(r.cos) |
                         reinterpret_cast<uintptr_t>(r.sin) | reinterpret_cast<uintptr_t>(r.k_out) | reinterpret_cast<uintptr_t>(r.v_out);
    const int64_t strides = r.k_stride_b | r.k_stride_h | r.k_stride_s | (r.v ? r.v_stride_b | r.v_stride_h | r.v_stride_s : 0) |
                            (r.cos ? r.cs_stride_b : 0) | r.o_stride_b | r.o_stride_h | r.o_stride_s;
    const int64_t chunks = (int64_t)r.batch * r.tokens * (r.dim / 16);
    if (!(at & 15) && !(strides & 7) && r.dim % 16 == 0 && r.width % 8 == 0 && chunks * r.heads < (1LL << 31)) {
        // four heads to a thread once that still gives every SM 1024 threads
        const int hpt = chunks * r.heads >= 4LL * kSmCount * 1024 ? 4 : 1;
        const unsigned items = (unsigned)(chunks * ((r.heads + hpt - 1) / hpt));
        if (r.is_bf16) rows_kernel<__nv_bfloat16><<<(items + 255) / 256, 256, 0, st>>>(r, hpt, items);
        else rows_kernel<__half><<<(items + 255) / 256, 256, 0, st>>>(r, hpt, items);
    } else {
        dim3 grid(r.tokens, r.heads, r.batch);
        if (r.is_bf16) rows_scalar_kernel<__nv_bfloat16><<<grid, 128, 0, st>>>(r);
        else rows_scalar_kernel<__half><<<grid, 128, 0, st>>>(r);
    }
    return cudaGetLastError() == cudaSuccess ? kOk : kCudaError;
}

int launch_dequantize(const DequantArgs& q, cudaStream_t st) {
    if (q.batch < 0 || q.heads <= 0 || q.tokens < 0 || q.block <= 0) return kBadArgument;
    if (q.mode < 0 || q.mode > 3) return kUnsupported;
    if ((int64_t)q.batch * q.tokens == 0) return kOk;
    if (!q.codes || !q.scale || !q.zero || !q.out) return kBadArgument;
    dim3 grid(q.tokens, q.heads, q.batch);
    if (q.is_bf16) { if (q.high_precision_zero) dequant_kernel<__nv_bfloat16, true><<<grid, 128, 0, st>>>(q); else dequant_kernel<__nv_bfloat16, false><<<grid, 128, 0, st>>>(q); }
    else           { if (q.high_precision_zero) dequant_kernel<__half, true><<<grid, 128, 0, st>>>(q); else dequant_kernel<__half, false><<<grid, 128, 0, st>>>(q); }
    return cudaGetLastError() == cudaSuccess ? kOk : kCudaError;
}

}  // namespace pkv
