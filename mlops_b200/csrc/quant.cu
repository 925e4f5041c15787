// HBM-bound row kernels around the grouped GEMMs: E4M3 quantisation of activation rows
// (optionally gathered into expert order), SwiGLU fused with the quantisation of its
// result, the routed SwiGLU backward, and the 128x128 weight-block quantiser.
//
// Scale equations (bit-reproducible on a CPU):
//   activation rows / 1x128 blocks: scale = max(amax * fp32(1/448), 1e-12)
//        (reference: src/mlops/kernels/quack_moe/quantize_rows.py:34-41)
//   weight 128x128 blocks:          scale = max(amax / 448, 1e-12)   (RN division)
//        (reference: src/mlops/kernels/block_fp8.py:48-60)
//   value: q = e4m3_rn(clamp(x / scale, -448, 448)) with an RN fp32 division.
//
// One warp owns one row; every lane moves 16 bytes per access, so a warp reads 512
// contiguous bytes of bf16 and writes 256 contiguous bytes of E4M3 per step.  A 128-wide
// scale block is the business of one half warp (16 lanes x 8 values).
#include "common.cuh"
#include "host_util.h"

namespace b200 {

constexpr int kRowWarps = 8;

__device__ __forceinline__ float halfwarp_max(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ uint4 pack8_bf16(const float (&v)[8]) {
  uint4 o;
  o.x = pack_bf16x2(v[0], v[1]);
  o.y = pack_bf16x2(v[2], v[3]);
  o.z = pack_bf16x2(v[4], v[5]);
  o.w = pack_bf16x2(v[6], v[7]);
  return o;
}

// mode 0: one scale per 128-column block.  mode 1: one scale per row (two passes).
__global__ void __launch_bounds__(kRowWarps * 32)
quantize_rows_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, long long src_rows,
                     const int* __restrict__ gather, int gather_div, long long rows, int D,
                     uint8_t* __restrict__ q, long long ldq, float* __restrict__ scales, long long s_row,
                     long long s_kb, int mode, __nv_bfloat16* __restrict__ copy, long long ldc, int* status) {
  const int lane = threadIdx.x & 31;
  const long long r = (long long)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (r >= rows) return;
  long long src = gather != nullptr ? (long long)(gather[r] / gather_div) : r;
  if (src < 0 || src >= src_rows) {  // a bad index is reported and reads row 0, never out of bounds
    if (lane == 0) report_error(status, ERR_BAD_OFFSETS, 20, (int)r);
    src = 0;
  }
  const __nv_bfloat16* xr = x + src * ldx;
  uint8_t* qr = q + r * ldq;
  if (mode == 0) {
    // two 256-column steps per iteration: both loads are in flight before either is used
    for (int c0 = 0; c0 < D; c0 += 512) {
      const int ca = c0 + lane * 8, cb = ca + 256;
      uint4 raw_a = make_uint4(0, 0, 0, 0), raw_b = make_uint4(0, 0, 0, 0);
      if (ca < D) raw_a = *reinterpret_cast<const uint4*>(xr + ca);
      if (cb < D) raw_b = *reinterpret_cast<const uint4*>(xr + cb);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = h == 0 ? ca : cb;
        float v[8];
        unpack8(h == 0 ? raw_a : raw_b, v);
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
        amax = halfwarp_max(amax);
        const float scale = fmaxf(amax * kInv448, 1e-12f);
        if (c < D) {
          *reinterpret_cast<uint2*>(qr + c) = quantize8(v, scale);
          if ((lane & 15) == 0) scales[r * s_row + (long long)(c >> 7) * s_kb] = scale;
          if (copy != nullptr) *reinterpret_cast<uint4*>(copy + r * ldc + c) = h == 0 ? raw_a : raw_b;
        }
      }
    }
  } else {
    float amax = 0.f;
    for (int c = lane * 8; c < D; c += 256) {
      float v[8];
      unpack8(*reinterpret_cast<const uint4*>(xr + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    }
    amax = warp_max(amax);
    const float scale = fmaxf(amax * kInv448, 1e-12f);
    for (int c = lane * 8; c < D; c += 256) {
      float v[8];
      unpack8(*reinterpret_cast<const uint4*>(xr + c), v);
      *reinterpret_cast<uint2*>(qr + c) = quantize8(v, scale);
    }
    if (lane == 0) scales[r * s_row] = scale;
  }
}

// The same quantisation, token-major: every token row is read and quantised ONCE and the
// result is written to each of the `fanout` output rows `slots[t * fanout + k]` (the
// expert-ordered rows of the token's assignments), instead of once per output row.  Same bytes
// and scales as quantize_rows_kernel with gather = order / fanout; 1/fanout of its arithmetic
// and source reads, so the pass is bound by its writes.  1x128 scales only.
//
// One warp per token and 512 columns, 16 columns per lane (a 128-column block is 8 lanes): every
// store moves 16 bytes per lane, nothing is carried from one piece of a row to the next, and a
// decode batch of 64 tokens still fills the machine.  Measured with eight slots a token, one warp
// per token -> now: 64 x 7168 38 -> 4.5 us, 3001 x 2048 18.8 -> 13.1, 8192 x 7168 150 -> 118 (5.1 TB/s).
__global__ void __launch_bounds__(kRowWarps * 32)
quantize_scatter_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, long long tokens, int chunks,
                        const int* __restrict__ slots, int fanout, long long rows_out, int D,
                        uint8_t* __restrict__ q, long long ldq, float* __restrict__ scales,
                        long long s_row, long long s_kb, __nv_bfloat16* __restrict__ copy, long long ldc,
                        int wide, int* status) {
  const int lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  const long long t = w / chunks;
  if (t >= tokens) return;
  const int chunk = (int)(w - t * chunks);
  const int c = chunk * 512 + lane * 16;
  const bool has_a = c < D, has_b = c + 8 < D;  // rows are a multiple of 8 columns
  const __nv_bfloat16* xr = x + t * ldx + c;
  uint4 raw_a = make_uint4(0, 0, 0, 0), raw_b = raw_a;
  if (has_a) raw_a = *reinterpret_cast<const uint4*>(xr);
  if (has_b) raw_b = *reinterpret_cast<const uint4*>(xr + 8);
  // lane k < fanout holds destination k; a slot outside the output is reported and skipped
  int mine = -1;
  if (lane < fanout) {
    mine = slots[t * fanout + lane];
    if (mine < 0 || mine >= rows_out) {
      if (chunk == 0) report_error(status, ERR_BAD_OFFSETS, 24, (int)t);
      mine = -1;
    }
  }
  float va[8], vb[8];
  unpack8(raw_a, va);
  unpack8(raw_b, vb);
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fmaxf(fabsf(va[i]), fabsf(vb[i])));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = fmaxf(amax * kInv448, 1e-12f);
  const uint2 qa = quantize8(va, scale), qb = quantize8(vb, scale);
  uint8_t* q_at = q + c;
  float* s_at = scales + (long long)(c >> 7) * s_kb;
  __nv_bfloat16* copy_at = copy + c;
#pragma unroll 4
  for (int k = 0; k < fanout; ++k) {
    const long long dst = __shfl_sync(0xffffffffu, mine, k);
    if (dst < 0 || !has_a) continue;
    if (wide && has_b) {
      *reinterpret_cast<uint4*>(q_at + dst * ldq) = make_uint4(qa.x, qa.y, qb.x, qb.y);
    } else {
      *reinterpret_cast<uint2*>(q_at + dst * ldq) = qa;
      if (has_b) *reinterpret_cast<uint2*>(q_at + dst * ldq + 8) = qb;
    }
    if ((lane & 7) == 0) s_at[dst * s_row] = scale;
    if (copy != nullptr) {
      *reinterpret_cast<uint4*>(copy_at + dst * ldc) = raw_a;
      if (has_b) *reinterpret_cast<uint4*>(copy_at + dst * ldc + 8) = raw_b;
    }
  }
}

// act = silu(gate) * up computed in fp32 from h13 = [gate | up] (each F wide), rounded
// once: to E4M3 with 1x128 scales (act_q / scales) and, when act_bf16 is given, to bf16.
// Optional GLM clamp: gate capped at `limit`, up clipped to [-limit, limit].
// One warp per `per_warp` consecutive pieces of 256 columns of a row: the next piece is loaded
// while one is worked on.  Issue-bound in its arithmetic: with the library's rounded reciprocal and scalar
// arithmetic 32768 rows of F = 14336 took 0.61 ms, with sigmoid8 and packed arithmetic 0.475 (5.0 TB/s);
// 512 rows of F = 2048 take 4.1 us instead of 10.
template <bool LIMITED>
__global__ void __launch_bounds__(kRowWarps * 32)
swiglu_quant_kernel(const __nv_bfloat16* __restrict__ h13, long long ldh, long long rows, int F,
                    uint8_t* __restrict__ act_q, long long ldq, float* __restrict__ scales,
                    long long s_row, long long s_kb, __nv_bfloat16* __restrict__ act_bf16,
                    long long lda, float limit, int per_warp, int warps_per_row) {
  const int lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  const long long r = w / warps_per_row;
  if (r >= rows) return;
  const int c_begin = (int)(w - r * warps_per_row) * per_warp * 256;
  const int c_end = min(F, c_begin + per_warp * 256);
  const __nv_bfloat16* hr = h13 + r * ldh;
  uint4 rg, ru;
  auto fetch = [&](int c) {
    rg = ru = make_uint4(0, 0, 0, 0);
    if (c < c_end) {
      rg = *reinterpret_cast<const uint4*>(hr + c);
      ru = *reinterpret_cast<const uint4*>(hr + F + c);
    }
  };
  fetch(c_begin + lane * 8);
  for (int c = c_begin + lane * 8; c - lane * 8 < c_end; c += 256) {
    float g[8], u[8], a[8], sig[8];
    unpack8(rg, g);
    unpack8(ru, u);
    fetch(c + 256);
    if constexpr (LIMITED) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        g[i] = fminf(g[i], limit);
        u[i] = fminf(fmaxf(u[i], -limit), limit);
      }
    }
    sigmoid8(g, sig);
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const Float2 silu = mul2(pack2(g[i], g[i + 1]), pack2(sig[i], sig[i + 1]));
      unpack2(mul2(silu, pack2(u[i], u[i + 1])), a[i], a[i + 1]);
      amax = fmaxf(amax, fmaxf(fabsf(a[i]), fabsf(a[i + 1])));
    }
    amax = halfwarp_max(amax);
    const float scale = fmaxf(amax * kInv448, 1e-12f);
    if (c < F) {
      if (act_q != nullptr) {
        *reinterpret_cast<uint2*>(act_q + r * ldq + c) = quantize8(a, scale);
        if ((lane & 15) == 0) scales[r * s_row + (long long)(c >> 7) * s_kb] = scale;
      }
      if (act_bf16 != nullptr) *reinterpret_cast<uint4*>(act_bf16 + r * lda + c) = pack8_bf16(a);
    }
  }
}

// Routed SwiGLU backward in one pass over h13 and r (= dy_row @ W2, before the route
// weight).  With score = route weight of the row:
//   dscore[row]  = <r, act>
//   g            = score * r
//   dgate        = g * up * (sig + silu * (1 - sig)),  dup = g * silu
//   grad_h13     = [dgate | dup]  -> E4M3 with 1x128 scales (and bf16 when asked)
//   act_scaled   = score * act    (bf16; operand of the down weight's gradient)
// (reference: src/mlops/kernels/quack_moe/swiglu_rows.py:100-199)
// gh_bf16 may alias h13 (the gradient written over the saved pre-activation): each thread reads
// the sixteen h13 values of an iteration before it stores the sixteen gradients to the same
// addresses, and no other thread touches them; act_scaled may alias r in the same way.
// One warp per row (the dot product stays in the warp); the next 256 columns are loaded while
// these are worked on.  32768 rows of F = 14336 with every output: 1.10 ms (6.0 TB/s); 1.36 ms with
// scalar arithmetic, which kept the kernel issue-bound.  Three blocks to an SM need 80 registers a
// thread; at the 83 the compiler takes unasked two fit, and the same took 1.20 ms.  (With a limit 80
// would spill.)
template <bool LIMITED>
__global__ void __launch_bounds__(kRowWarps * 32, LIMITED ? 2 : 3)
dswiglu_routed_kernel(const __nv_bfloat16* h13, long long ldh,  // may be the same buffer as gh_bf16
                      const __nv_bfloat16* rmat, long long ldr,       // may be the same buffer as act_scaled
                      const float* __restrict__ route_weights, long long n_weights,
                      const int* __restrict__ order, long long rows, int F, float* __restrict__ dscore,
                      uint8_t* __restrict__ gh_q, long long ldq, float* __restrict__ gh_scales,
                      long long s_row, long long s_kb, __nv_bfloat16* gh_bf16,
                      long long ldg, __nv_bfloat16* act_scaled, long long lda, float limit,
                      int* status) {
  const int lane = threadIdx.x & 31;
  const long long r = (long long)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (r >= rows) return;
  const __nv_bfloat16* hr = h13 + r * ldh;
  const __nv_bfloat16* rr = rmat + r * ldr;
  uint4 rg, ru, rx;
  auto fetch = [&](int c) {
    rg = ru = rx = make_uint4(0, 0, 0, 0);
    if (c < F) {
      rg = *reinterpret_cast<const uint4*>(hr + c);
      ru = *reinterpret_cast<const uint4*>(hr + F + c);
      rx = *reinterpret_cast<const uint4*>(rr + c);
    }
  };
  fetch(lane * 8);
  long long which = order[r];
  if (which < 0 || which >= n_weights) {
    if (lane == 0) report_error(status, ERR_BAD_OFFSETS, 21, (int)r);
    which = 0;
  }
  const Float2 score = splat2(route_weights[which]);
  const Float2 one = splat2(1.0f), minus_one = splat2(-1.0f);
  float dot = 0.f;
  for (int c0 = 0; c0 < F; c0 += 256) {
    const int c = c0 + lane * 8;
    float g[8], u[8], rv[8], dg[8], du[8], sig[8];
    uint32_t scaled[4];  // score * act
    unpack8(rg, g);
    unpack8(ru, u);
    unpack8(rx, rv);
    fetch(c + 256);
    uint32_t keep_g = 0xff, keep_u = 0xff;
    if constexpr (LIMITED) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (!(g[i] <= limit)) keep_g &= ~(1u << i);
        if (!(u[i] >= -limit && u[i] <= limit)) keep_u &= ~(1u << i);
        g[i] = fminf(g[i], limit);
        u[i] = fminf(fmaxf(u[i], -limit), limit);
      }
    }
    sigmoid8(g, sig);
    float amax_g = 0.f, amax_u = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const Float2 s2 = pack2(sig[i], sig[i + 1]), u2 = pack2(u[i], u[i + 1]), r2 = pack2(rv[i], rv[i + 1]);
      const Float2 silu = mul2(pack2(g[i], g[i + 1]), s2);
      const Float2 act = mul2(silu, u2);
      float act0, act1;
      unpack2(act, act0, act1);
      dot = fmaf(rv[i + 1], act1, fmaf(rv[i], act0, dot));  // one sum in column order
      const Float2 go = mul2(score, r2);
      const Float2 slope = mad2(silu, mad2(s2, minus_one, one), s2);  // sig + silu (1 - sig)
      unpack2(mul2(mul2(go, u2), slope), dg[i], dg[i + 1]);
      unpack2(mul2(go, silu), du[i], du[i + 1]);
      unpack2(mul2(score, act), act0, act1);
      scaled[i / 2] = pack_bf16x2(act0, act1);
      if constexpr (LIMITED) {
#pragma unroll
        for (int h = i; h < i + 2; ++h) {
          if (!((keep_g >> h) & 1)) dg[h] = 0.f;
          if (!((keep_u >> h) & 1)) du[h] = 0.f;
        }
      }
      amax_g = fmaxf(amax_g, fmaxf(fabsf(dg[i]), fabsf(dg[i + 1])));
      amax_u = fmaxf(amax_u, fmaxf(fabsf(du[i]), fabsf(du[i + 1])));
    }
    amax_g = halfwarp_max(amax_g);
    amax_u = halfwarp_max(amax_u);
    if (c < F) {
      if (gh_q != nullptr) {
        const float sg = fmaxf(amax_g * kInv448, 1e-12f);
        const float su = fmaxf(amax_u * kInv448, 1e-12f);
        *reinterpret_cast<uint2*>(gh_q + r * ldq + c) = quantize8(dg, sg);
        *reinterpret_cast<uint2*>(gh_q + r * ldq + F + c) = quantize8(du, su);
        if ((lane & 15) == 0) {
          gh_scales[r * s_row + (long long)(c >> 7) * s_kb] = sg;
          gh_scales[r * s_row + (long long)((F + c) >> 7) * s_kb] = su;
        }
      }
      if (gh_bf16 != nullptr) {
        *reinterpret_cast<uint4*>(gh_bf16 + r * ldg + c) = pack8_bf16(dg);
        *reinterpret_cast<uint4*>(gh_bf16 + r * ldg + F + c) = pack8_bf16(du);
      }
      if (act_scaled != nullptr)
        *reinterpret_cast<uint4*>(act_scaled + r * lda + c) = make_uint4(scaled[0], scaled[1], scaled[2], scaled[3]);
    }
  }
  dot = warp_sum(dot);
  if (lane == 0 && dscore != nullptr) dscore[r] = dot;
}

// One CTA per 128x128 block of a [E, out, in] weight (bf16 or fp32 source), read ONCE: 512 threads
// hold the block in registers (32 values each) between the maximum and the cast.  16-byte loads: a
// warp's access is one fp32 row of the block or two bf16 rows; stores of 4 bytes (fp32) or 8 bytes
// (bf16) per lane fill whole 128-byte lines.  Needs rows whose length is a multiple of the vector
// and 16-byte aligned sources; quantize_blocks_general_kernel serves the rest.  Bound by HBM (5
// bytes a value from fp32): both weights of 128 experts with D = 2048, F = 768, 3.0 GB in all, take
// 0.50 ms (6.0 TB/s); two passes of 4-byte loads and byte stores took 0.82 ms.
template <typename SrcT>
__global__ void __launch_bounds__(512, 2)
quantize_blocks_kernel(const SrcT* __restrict__ w, int out, int in, int blocks_out, int blocks_in,
                       uint8_t* __restrict__ q, float* __restrict__ scale) {
  constexpr int kVec = 16 / sizeof(SrcT);   // values per load
  constexpr int kLanes = 128 / kVec;        // lanes per row
  constexpr int kRows = 512 / kLanes;       // rows per pass
  constexpr int kPasses = 128 / kRows;
  __shared__ uint32_t red[16];
  const long long e = blockIdx.z;
  const int br = blockIdx.y, bc = blockIdx.x;
  const int row0 = br * 128 + threadIdx.x / kLanes;
  const int col = bc * 128 + (threadIdx.x % kLanes) * kVec;
  const SrcT* base = w + e * (long long)out * in + col;
  uint4 raw[kPasses];
#pragma unroll
  for (int i = 0; i < kPasses; ++i) {
    const int row = row0 + i * kRows;
    raw[i] = make_uint4(0, 0, 0, 0);
    if (row < out && col < in) raw[i] = __ldcs(reinterpret_cast<const uint4*>(base + (long long)row * in));
  }
  auto value = [&](int i, int k) {
    const uint32_t word[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
    if constexpr (sizeof(SrcT) == 4) return __uint_as_float(word[k]);
    else return __uint_as_float((k & 1) ? (word[k >> 1] & 0xffff0000u) : (word[k >> 1] << 16));
  };
  // the maximum over the bit patterns of |x|: non-negative floats order like their bits, and an
  // infinity or a NaN shows as a pattern of at least 0x7f800000
  uint32_t top = 0;
#pragma unroll
  for (int i = 0; i < kPasses; ++i)
#pragma unroll
    for (int k = 0; k < kVec; ++k) top = max(top, __float_as_uint(value(i, k)) & 0x7fffffffu);
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = top;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 16; ++i) top = max(top, red[i]);
  const bool finite = top < 0x7f800000u;
  if (!finite) {  // a NaN does not count towards the maximum
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < kPasses; ++i)
#pragma unroll
      for (int k = 0; k < kVec; ++k) amax = fmaxf(amax, fabsf(value(i, k)));
    top = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
    __syncthreads();  // everyone has read the first maximum
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = top;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 16; ++i) top = max(top, red[i]);
  }
  const float s = fmaxf(__fdiv_rn(__uint_as_float(top), 448.0f), 1e-12f);
  if (threadIdx.x == 0) scale[(e * blocks_out + br) * blocks_in + bc] = s;
  const float inv = __frcp_rn(s);
  uint8_t* qbase = q + e * (long long)out * in + col;
#pragma unroll
  for (int i = 0; i < kPasses; ++i) {
    const int row = row0 + i * kRows;
    uint32_t packed[kVec / 4];
    // the exact-division shortcut of quantize8; blocks with an infinity or a NaN always divide
    bool exact = finite;
#pragma unroll
    for (int k = 0; k < kVec; k += 2) {
      const float q0 = value(i, k) * inv, q1 = value(i, k + 1) * inv;
      const float e0 = q0 * 4.76837158203125e-7f, e1 = q1 * 4.76837158203125e-7f;  // 2^-21
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(q0 + e0, q1 + e1), __NV_SATFINITE, __NV_E4M3);
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(q0 - e0, q1 - e1), __NV_SATFINITE, __NV_E4M3);
      exact = exact && (hi == lo);
      packed[k >> 2] = (k & 2) ? packed[k >> 2] | (hi << 16) : hi;
    }
    if (!exact) {
#pragma unroll
      for (int k = 0; k < kVec; ++k) {
        const uint32_t byte = (uint32_t)to_e4m3(__fdiv_rn(value(i, k), s)) << (8 * (k & 3));
        packed[k >> 2] = (k & 3) ? packed[k >> 2] | byte : byte;
      }
    }
    if (row < out && col < in) {
      uint8_t* at = qbase + (long long)row * in;
      if constexpr (kVec == 4) *reinterpret_cast<uint32_t*>(at) = packed[0];
      else *reinterpret_cast<uint2*>(at) = make_uint2(packed[0], packed[kVec / 4 - 1]);
    }
  }
}

// The same for rows of any length and alignment: value by value, two passes.
template <typename SrcT>
__global__ void __launch_bounds__(256)
quantize_blocks_general_kernel(const SrcT* __restrict__ w, int out, int in, int blocks_out, int blocks_in,
                               uint8_t* __restrict__ q, float* __restrict__ scale) {
  __shared__ float red[8];
  const long long e = blockIdx.z;
  const int br = blockIdx.y, bc = blockIdx.x;
  const SrcT* base = w + e * (long long)out * in;
  uint8_t* qbase = q + e * (long long)out * in;
  const int tr = threadIdx.x >> 5;  // 8 row groups
  const int tc = threadIdx.x & 31;  // 32 column groups of 4
  float amax = 0.f;
  for (int rr = tr; rr < 128; rr += 8) {
    const int row = br * 128 + rr;
    if (row >= out) break;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int col = bc * 128 + tc * 4 + k;
      if (col < in) amax = fmaxf(amax, fabsf((float)base[(long long)row * in + col]));
    }
  }
  amax = warp_max(amax);
  if (tc == 0) red[tr] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
  const float s = fmaxf(__fdiv_rn(amax, 448.0f), 1e-12f);
  if (threadIdx.x == 0) scale[(e * blocks_out + br) * blocks_in + bc] = s;
  for (int rr = tr; rr < 128; rr += 8) {
    const int row = br * 128 + rr;
    if (row >= out) break;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int col = bc * 128 + tc * 4 + k;
      if (col < in) {
        qbase[(long long)row * in + col] = to_e4m3(__fdiv_rn((float)base[(long long)row * in + col], s));
      }
    }
  }
}


// ---------------------------------------------------------------------------------------
// Column-scaled E4M3 for the FP8 weight gradient: the rows of a group (an expert's tokens)
// share one scale per COLUMN, scale = max(amax over the group's rows * fp32(1/448), 1e-12),
// the row quantiser's equations applied to a column (reference: the per-feature scales of
// src/mlops/kernels/quack_moe/quantize_transpose.py:126-133).  The output stays token-major:
// the weight-gradient GEMM reads both operands MN-major, so no transpose is ever stored.
// `offsets` holds segments * groups + 1 row boundaries; range i belongs to group i % groups.
// Pass 1: column maxima of every 256-row x 256-column piece, merged with atomicMax on the bit
// pattern (non-negative floats order like their bits).  Pass 2: maxima -> scales in place.
// Pass 3: the cast.
// ---------------------------------------------------------------------------------------
constexpr int kColRows = 256;  // rows per block: 8 warps x 32 rows

// The range (index into offsets) that holds row r; ranges may be empty.
__device__ __forceinline__ int range_of_row(const int* __restrict__ offsets, int ranges, int r) {
  int lo = 0, hi = ranges;  // invariant: offsets[lo] <= r < offsets[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (offsets[mid] <= r) lo = mid;
    else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(256)
column_amax_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, int rows, int width,
                   const int* __restrict__ offsets, int groups, int segments, unsigned int* __restrict__ amax_bits) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.y * 256 + lane * 8;
  const int r0 = blockIdx.x * kColRows + warp * 32;
  if (c >= width || r0 >= rows) return;
  const int ranges = groups * segments;
  const int r_begin = max(r0, offsets[0]);                       // rows outside the table belong to no group
  const int r_end = min(min(r0 + 32, rows), offsets[ranges]);
  if (r_begin >= r_end) return;
  int range = range_of_row(offsets, ranges, r_begin);
  int range_end = offsets[range + 1];
  float m[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  auto flush = [&](int g) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (m[i] > 0.f) atomicMax(amax_bits + (long long)g * width + c + i, __float_as_uint(m[i]));
      m[i] = 0.f;
    }
  };
  for (int r = r_begin; r < r_end; ++r) {
    if (r >= range_end) {  // the row belongs to a later range: hand in what this one gathered
      flush(range % groups);
      range = range_of_row(offsets, ranges, r);
      range_end = offsets[range + 1];
    }
    float v[8];
    unpack8(*reinterpret_cast<const uint4*>(x + (long long)r * ldx + c), v);
#pragma unroll
    for (int i = 0; i < 8; ++i) m[i] = fmaxf(m[i], fabsf(v[i]));  // a NaN never wins: the scale stays finite
  }
  flush(range % groups);
}

__global__ void __launch_bounds__(256)
column_scale_kernel(float* __restrict__ scales, long long n) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i < n) scales[i] = fmaxf(scales[i] * kInv448, 1e-12f);  // the maxima arrive as fp32 bit patterns
}

__global__ void __launch_bounds__(256)
column_cast_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, int rows, int width,
                   const int* __restrict__ offsets, int groups, int segments, const float* __restrict__ scales,
                   uint8_t* __restrict__ q, long long ldq) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.y * 256 + lane * 8;
  const int r0 = blockIdx.x * kColRows + warp * 32;
  if (c >= width || r0 >= rows) return;
  const int ranges = groups * segments;
  const int r_begin = max(r0, offsets[0]);
  const int r_end = min(min(r0 + 32, rows), offsets[ranges]);
  int range = -1, range_end = -1;
  float sc[8], inv[8];
  for (int r = r_begin; r < r_end; ++r) {
    if (r >= range_end) {
      range = range_of_row(offsets, ranges, r);
      range_end = offsets[range + 1];
      const float* sg = scales + (long long)(range % groups) * width + c;
      const float4 a = *reinterpret_cast<const float4*>(sg), b = *reinterpret_cast<const float4*>(sg + 4);
      sc[0] = a.x; sc[1] = a.y; sc[2] = a.z; sc[3] = a.w;
      sc[4] = b.x; sc[5] = b.y; sc[6] = b.z; sc[7] = b.w;
#pragma unroll
      for (int i = 0; i < 8; ++i) inv[i] = __frcp_rn(sc[i]);
    }
    float v[8];
    unpack8(*reinterpret_cast<const uint4*>(x + (long long)r * ldx + c), v);
    // the same exact-division shortcut as quantize8, with one scale per value
    uint32_t w[2] = {0, 0};
    bool exact = true;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const float q0 = v[i] * inv[i], q1 = v[i + 1] * inv[i + 1];
      const float e0 = q0 * 4.76837158203125e-7f, e1 = q1 * 4.76837158203125e-7f;  // 2^-21
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(q0 + e0, q1 + e1), __NV_SATFINITE, __NV_E4M3);
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(q0 - e0, q1 - e1), __NV_SATFINITE, __NV_E4M3);
      exact = exact && (hi == lo);
      w[i >> 2] |= (hi & 0xffffu) << (8 * (i & 3));
    }
    if (!exact) {
      w[0] = w[1] = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        w[i >> 2] |= (uint32_t)to_e4m3(__fdiv_rn(v[i], sc[i])) << (8 * (i & 3));
      }
    }
    *reinterpret_cast<uint2*>(q + (long long)r * ldq + c) = make_uint2(w[0], w[1]);
  }
}

}  // namespace b200

using namespace b200;

static inline unsigned row_grid(long long rows) { return (unsigned)((rows + kRowWarps - 1) / kRowWarps); }

extern "C" int b200moe_quantize_rows(const void* x, long long ldx, long long src_rows, const int32_t* gather,
                                     int gather_div, long long rows, int width, void* q, long long ldq,
                                     float* scales, long long scale_row_stride, long long scale_block_stride,
                                     int mode, void* copy, long long ldc, int32_t* status, void* stream) {
  if (!x || !q || !scales || !status || rows < 0 || width <= 0 || (mode != 0 && mode != 1)) return B200MOE_ERR_ARG;
  if (rows > 0 && (src_rows <= 0 || (gather == nullptr && src_rows < rows))) return B200MOE_ERR_ARG;
  if (copy != nullptr && (mode != 0 || (ldc % 8) || ((uintptr_t)copy & 15))) return B200MOE_ERR_ARG;
  if (gather != nullptr && gather_div <= 0) return B200MOE_ERR_ARG;
  if ((width % 8) || (ldx % 8) || (ldq % 8) || ((uintptr_t)x & 15) || ((uintptr_t)q & 7))
    return B200MOE_ERR_ALIGN;
  if (rows == 0) return B200MOE_OK;
  quantize_rows_kernel<<<row_grid(rows), kRowWarps * 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(x), ldx, src_rows, gather, gather_div > 0 ? gather_div : 1, rows,
      width, reinterpret_cast<uint8_t*>(q), ldq, scales, scale_row_stride, scale_block_stride, mode,
      reinterpret_cast<__nv_bfloat16*>(copy), ldc, status);
  return launch_status();
}

extern "C" int b200moe_quantize_rows_scatter(const void* x, long long ldx, long long tokens, const int32_t* slots,
                                             int fanout, long long rows_out, int width, void* q, long long ldq,
                                             float* scales, long long scale_row_stride,
                                             long long scale_block_stride, void* copy, long long ldc,
                                             int32_t* status, void* stream) {
  if (!x || !slots || !q || !scales || !status || tokens < 0 || rows_out < 0 || width <= 0) return B200MOE_ERR_ARG;
  if (fanout <= 0 || fanout > 32) return B200MOE_ERR_LIMIT;
  if (copy != nullptr && ((ldc % 8) || ((uintptr_t)copy & 15))) return B200MOE_ERR_ALIGN;
  if ((width % 8) || (ldx % 8) || (ldq % 8) || ((uintptr_t)x & 15) || ((uintptr_t)q & 7))
    return B200MOE_ERR_ALIGN;
  if (tokens == 0) return B200MOE_OK;
  const int chunks = (width + 511) / 512;
  const int wide = (ldq % 16) == 0 && ((uintptr_t)q & 15) == 0;
  quantize_scatter_kernel<<<row_grid(tokens * chunks), kRowWarps * 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(x), ldx, tokens, chunks, slots, fanout, rows_out, width,
      reinterpret_cast<uint8_t*>(q), ldq, scales, scale_row_stride, scale_block_stride,
      reinterpret_cast<__nv_bfloat16*>(copy), ldc, wide, status);
  return launch_status();
}

extern "C" int b200moe_swiglu_quantize(const void* h13, long long ldh, long long rows, int width,
                                       void* act_q, long long ldq, float* scales,
                                       long long scale_row_stride, long long scale_block_stride,
                                       void* act_bf16, long long lda, float limit, int limited,
                                       void* stream) {
  if (!h13 || rows < 0 || width <= 0 || (!act_q && !act_bf16) || (act_q && !scales)) return B200MOE_ERR_ARG;
  if ((width % 8) || (ldh % 8) || (ldq % 8) || (lda % 8) || ((uintptr_t)h13 & 15) || ((uintptr_t)act_q & 7) ||
      ((uintptr_t)act_bf16 & 15))
    return B200MOE_ERR_ALIGN;
  if (rows == 0) return B200MOE_OK;
  // a warp per row where that gives every SM 32 warps, a warp per 256 columns where it does not
  const int chunks = (width + 255) / 256;
  const int per_warp = rows >= 32LL * sm_count_device() ? chunks : 1;
  const int warps_per_row = (chunks + per_warp - 1) / per_warp;
  auto kern = limited ? swiglu_quant_kernel<true> : swiglu_quant_kernel<false>;
  kern<<<row_grid(rows * warps_per_row), kRowWarps * 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(h13), ldh, rows, width, reinterpret_cast<uint8_t*>(act_q), ldq, scales,
      scale_row_stride, scale_block_stride, reinterpret_cast<__nv_bfloat16*>(act_bf16), lda, limit, per_warp,
      warps_per_row);
  return launch_status();
}

extern "C" int b200moe_dswiglu_routed(const void* h13, long long ldh, const void* r, long long ldr,
                                      const float* route_weights, long long n_weights, const int32_t* order,
                                      long long rows, int width, float* dscore, void* grad_h13_q, long long ldq,
                                      float* grad_h13_scales, long long scale_row_stride,
                                      long long scale_block_stride, void* grad_h13_bf16, long long ldg,
                                      void* act_scaled, long long lda, float limit, int limited,
                                      int32_t* status, void* stream) {
  if (!h13 || !r || !route_weights || !order || !status || rows < 0 || width <= 0) return B200MOE_ERR_ARG;
  if (rows > 0 && n_weights <= 0) return B200MOE_ERR_ARG;
  if (grad_h13_q && !grad_h13_scales) return B200MOE_ERR_ARG;
  if ((width % 8) || (ldh % 8) || (ldr % 8) || (ldq % 8) || (ldg % 8) || (lda % 8)) return B200MOE_ERR_ALIGN;
  if (((uintptr_t)h13 & 15) || ((uintptr_t)r & 15) || ((uintptr_t)grad_h13_q & 7) ||
      ((uintptr_t)grad_h13_bf16 & 15) || ((uintptr_t)act_scaled & 15))
    return B200MOE_ERR_ALIGN;
  if (rows == 0) return B200MOE_OK;
  auto kern = limited ? dswiglu_routed_kernel<true> : dswiglu_routed_kernel<false>;
  kern<<<row_grid(rows), kRowWarps * 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(h13), ldh, reinterpret_cast<const __nv_bfloat16*>(r), ldr,
      route_weights, n_weights, order, rows, width, dscore, reinterpret_cast<uint8_t*>(grad_h13_q), ldq,
      grad_h13_scales, scale_row_stride, scale_block_stride, reinterpret_cast<__nv_bfloat16*>(grad_h13_bf16), ldg,
      reinterpret_cast<__nv_bfloat16*>(act_scaled), lda, limit, status);
  return launch_status();
}

// E4M3 rows of x [rows, width] with one scale per (group, column): scales [groups, width].
// Rows outside every range (none, when offsets[0] == 0 and the last entry == rows) are not written.
extern "C" int b200moe_quantize_columns(const void* x, long long ldx, long long rows, int width,
                                        const int32_t* offsets, int groups, int segments, void* q, long long ldq,
                                        float* scales, void* stream) {
  if (!x || !offsets || !q || !scales || rows < 0 || width <= 0 || groups <= 0 || segments <= 0)
    return B200MOE_ERR_ARG;
  if (rows > 0x7fffffffLL) return B200MOE_ERR_LIMIT;
  if ((width % 8) || (ldx % 8) || (ldq % 8) || ((uintptr_t)x & 15) || ((uintptr_t)q & 7) || ((uintptr_t)scales & 15))
    return B200MOE_ERR_ALIGN;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const long long n = (long long)groups * width;
  if (cudaMemsetAsync(scales, 0, (size_t)n * sizeof(float), s) != cudaSuccess) return B200MOE_ERR_LAUNCH;
  if (rows > 0) {
    dim3 grid((unsigned)((rows + kColRows - 1) / kColRows), (unsigned)((width + 255) / 256));
    column_amax_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), ldx, (int)rows, width,
                                            offsets, groups, segments, reinterpret_cast<unsigned int*>(scales));
  }
  column_scale_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(scales, n);
  if (rows > 0) {
    dim3 grid((unsigned)((rows + kColRows - 1) / kColRows), (unsigned)((width + 255) / 256));
    column_cast_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), ldx, (int)rows, width,
                                            offsets, groups, segments, scales, reinterpret_cast<uint8_t*>(q), ldq);
  }
  return launch_status();
}


template <typename SrcT>
static void launch_quantize_blocks(dim3 grid, const void* w, int out, int in, void* q, float* scale, cudaStream_t s) {
  constexpr int kVec = 16 / sizeof(SrcT);
  const SrcT* src = reinterpret_cast<const SrcT*>(w);
  uint8_t* dst = reinterpret_cast<uint8_t*>(q);
  if (in % kVec == 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)q % kVec) == 0)
    quantize_blocks_kernel<SrcT><<<grid, 512, 0, s>>>(src, out, in, grid.y, grid.x, dst, scale);
  else
    quantize_blocks_general_kernel<SrcT><<<grid, 256, 0, s>>>(src, out, in, grid.y, grid.x, dst, scale);
}

extern "C" int b200moe_quantize_blocks(const void* w, int src_is_fp32, int experts, int out, int in,
                                       void* q, float* scale, void* stream) {
  if (!w || !q || !scale || experts <= 0 || out <= 0 || in <= 0) return B200MOE_ERR_ARG;
  if (experts > 65535) return B200MOE_ERR_LIMIT;
  const int bo = (out + 127) / 128, bi = (in + 127) / 128;
  if (bo > 65535) return B200MOE_ERR_LIMIT;
  dim3 grid(bi, bo, experts);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (src_is_fp32) launch_quantize_blocks<float>(grid, w, out, in, q, scale, s);
  else launch_quantize_blocks<__nv_bfloat16>(grid, w, out, in, q, scale, s);
  return launch_status();
}
