// Device helpers shared by the sm_100a kernels: the INT8 code rule, bf16/fp16 row I/O, the in-register
// Walsh-Hadamard butterfly and the warp-level MMA wrappers.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/linquant_b200.h"

namespace lq {

// ---- host-side error plumbing (defined in lq_api.cu)
int fail(int status, const char* fmt, ...);
int check_launch(const char* what);
int sm_count();  // of the current device

// ---- programmatic dependent launch
// The kernels of a call form a chain in which each reads what the one before wrote. They are launched with the
// stream-serialisation attribute and open with pdl_enter(), which waits until everything before has completed and is
// visible: the launch itself (block scheduling, instruction and parameter fetch) then overlaps the end of the kernel before,
// 1 to 3 us per kernel, which is a third of a short prompt's time (a Mamba-2 layer on one chunk: 55 -> 38 us). All
// memory traffic, barrier set-up and tensor-memory allocation stay behind the wait. No kernel triggers its successor
// early: CTAs that are placed while a kernel is still running fill whatever SMs have room, several to an SM, and the serial
// state passes then keep that uneven placement to their end (DeltaNet, 1 x 1024 tokens: 75 us instead of 60).
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}
template <typename... KArgs, typename... Args>
static inline cudaError_t launch(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}
// More than 48 KB of dynamic shared memory: the opt-in is set on every launch (it is per kernel and device and costs a
// fraction of a microsecond).
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_opt_in(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return e != cudaSuccess ? e : launch(kern, grid, block, smem, st, args...);
}

// ---- the code rule (zoo/simple_gla.py:16-20; invariances.py:91-100)
// y = x * inv (fp32, its own rounding), half away from zero, clamp to +-qmax. Clamping first and truncating
// y + copysign(0.5, y) afterwards gives the same integer for every finite y.
__device__ __forceinline__ int q8(float x, float inv, float qmax) {
  float y = __fmul_rn(x, inv);
  y = fminf(fmaxf(y, -qmax), qmax);
  return __float2int_rz(__fadd_rn(y, copysignf(0.5f, y)));
}

// Four codes on the +-127 grid, packed: the lower clamp by hand, the upper one by the saturating pack (a value above
// 127.5 truncates to >= 127 and saturates to 127). Same codes as q8(x, inv, 127) four times and pack4.
__device__ __forceinline__ uint32_t q8x4_127(float x0, float x1, float x2, float x3, float inv);

__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d) {
  uint32_t lo = __byte_perm((uint32_t)a, (uint32_t)b, 0x0040);
  uint32_t hi = __byte_perm((uint32_t)c, (uint32_t)d, 0x0040);
  return __byte_perm(lo, hi, 0x5410);
}

// two int32 codes -> two saturated INT8 in the low half of the result, `upper` shifted into the high half
// (cvt.pack.sat.s8.s32.b32 d, a, b, c:  d = sat8(a) << 8 | sat8(b) | c << 16)
__device__ __forceinline__ uint32_t pack_sat_s8x2(int hi, int lo, uint32_t upper) {
  uint32_t d;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;\n" : "=r"(d) : "r"(hi), "r"(lo), "r"(upper));
  return d;
}
__device__ __forceinline__ int q8_lower127(float x, float inv) {
  const float y = fmaxf(__fmul_rn(x, inv), -127.f);
  return __float2int_rz(__fadd_rn(y, copysignf(0.5f, y)));
}
__device__ __forceinline__ uint32_t q8x4_127(float x0, float x1, float x2, float x3, float inv) {
  return pack_sat_s8x2(q8_lower127(x1, inv), q8_lower127(x0, inv), pack_sat_s8x2(q8_lower127(x3, inv), q8_lower127(x2, inv), 0u));
}
// Byte I of w, where w holds four INT8 codes XOR 0x80 (code + 128 as an unsigned byte), as an exact float: the byte
// becomes the low mantissa bits of 2^23 and the offset is subtracted -- no trip through the conversion unit.
template <int I>
__device__ __forceinline__ float s8_to_float(uint32_t w_xor80) {
  return __fsub_rn(__uint_as_float(__byte_perm(w_xor80, 0x4B000000u, 0x7540 | I)), 8388736.0f);
}

// ---- row orders of the two tiles that are B operands of the output contractions
// The k_local tile and the stored-state tile are laid out so that MMA column n of the output kernel is simply row n
// of the tile, while a thread's accumulator fragment still covers four consecutive tokens (k_local) or eight
// consecutive value channels (state). Within each group the row index is a fixed bit permutation of the token /
// channel index.
__device__ __host__ __forceinline__ int kl_row_of_token(int t) {  // low 4 bits [j1 j0 h e] -> [h j1 j0 e]
  return (t & ~15) | (((t >> 1) & 1) << 3) | (((t >> 2) & 3) << 1) | (t & 1);
}
__device__ __host__ __forceinline__ int state_row_of_channel(int v) {  // low 5 bits [j1 j0 n1 n0 e] -> [n1 n0 j1 j0 e]
  return (v & ~31) | (((v >> 1) & 3) << 3) | (((v >> 3) & 3) << 1) | (v & 1);
}
// The w_read tile [C,K] is the B operand of the delta state pass: per 32-channel block, the 32-byte rows of the 64 tokens in
// MMA-column order (n-tile (t >> 1) & 7, column 2 (t >> 4) + (t & 1): a lane's accumulators are then sixteen consecutive
// tokens), so that a fragment load is 256 contiguous bytes.
__device__ __host__ __forceinline__ int wq_offset(int t, int k) {
  return (k >> 5) * 2048 + ((((t >> 1) & 7) << 3) | ((t >> 4) << 1) | (t & 1)) * 32 + (k & 31);
}

// ---- activation dtype traits
template <typename T>
struct Act;
template <>
struct Act<__half> {
  static __device__ __forceinline__ void unpack8(const uint4& r, float (&x)[8]) {
    const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __half22float2(h[i]);
      x[2 * i] = f.x;
      x[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ float round(float x) { return __half2float(__float2half_rn(x)); }
  static __device__ __forceinline__ __half from(float x) { return __float2half_rn(x); }
  static __device__ __forceinline__ float to(__half x) { return __half2float(x); }
  static __device__ __forceinline__ float get(uint32_t w, int hi) {  // one of the two values of a packed word
    return __half2float(__ushort_as_half((unsigned short)(hi ? w >> 16 : w & 0xffffu)));
  }
  static __device__ __forceinline__ uint32_t pack2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
};
template <>
struct Act<__nv_bfloat16> {
  static __device__ __forceinline__ void unpack8(const uint4& r, float (&x)[8]) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[2 * i] = __uint_as_float(w[i] << 16);
      x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  static __device__ __forceinline__ float round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
  static __device__ __forceinline__ __nv_bfloat16 from(float x) { return __float2bfloat16_rn(x); }
  static __device__ __forceinline__ float to(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ float get(uint32_t w, int hi) { return __uint_as_float(hi ? w & 0xffff0000u : w << 16); }
  static __device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
};
template <>
struct Act<float> {
  static __device__ __forceinline__ float round(float x) { return x; }
};

// ---- Walsh-Hadamard butterfly over a row of D = 8 * LPR values held 8 per lane by LPR consecutive lanes
// (lane-in-row r holds elements 8r .. 8r+7). Sylvester ordering, unnormalised.
template <int LPR>
__device__ __forceinline__ void fwht8(float (&x)[8], int r) {
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if ((i & s) == 0) {
        float a = x[i], b = x[i | s];
        x[i] = a + b;
        x[i | s] = a - b;
      }
    }
  }
#pragma unroll
  for (int m = 1; m < LPR; m <<= 1) {
    const float s = (r & m) ? -1.0f : 1.0f;  // upper half of the butterfly: other - x, lower: x + other (one fma, exact)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float other = __shfl_xor_sync(0xffffffffu, x[i], m);
      x[i] = fmaf(x[i], s, other);
    }
  }
}

// ---- warp MMA wrappers (row.col, A and B both with the reduction index contiguous)
__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// first product of an INT8 accumulator chain: C = 0 without zeroing registers
__device__ __forceinline__ void mma_s8_first(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// four INT8 codes in one word -> two half2 words (codes 0,1 and 2,3), exact: (c ^ 0x80) + 1024 - 1152
__device__ __forceinline__ void s8x4_to_h2x2(uint32_t w, uint32_t& h01, uint32_t& h23) {
  const uint32_t u = w ^ 0x80808080u;
  uint32_t a = __byte_perm(u, 0x64646464u, 0x4140);
  uint32_t b = __byte_perm(u, 0x64646464u, 0x4342);
  const __half2 bias = __half2half2(__ushort_as_half((unsigned short)0x6480));  // 1152.0
  __half2 ha = __hsub2(*reinterpret_cast<__half2*>(&a), bias);
  __half2 hb = __hsub2(*reinterpret_cast<__half2*>(&b), bias);
  h01 = *reinterpret_cast<uint32_t*>(&ha);
  h23 = *reinterpret_cast<uint32_t*>(&hb);
}

// two fp32 values in one register pair: one instruction for both (each rounded on its own, as the scalar forms)
struct F2 {
  unsigned long long v;
  __device__ __forceinline__ F2() {}
  __device__ __forceinline__ F2(float x, float y) { asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "f"(x), "f"(y)); }
  __device__ __forceinline__ void get(float& x, float& y) const { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(x), "=f"(y) : "l"(v)); }
};
__device__ __forceinline__ F2 mul2(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 add2(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }

__device__ __forceinline__ F2 sub2(F2 a, F2 b) { F2 r; asm("sub.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }

// e^x of two values as 2^(x log2 e), one hardware exponential each; a result below 2^-126 is zero (the non-flushing form takes
// three more instructions a value to keep it)
__device__ __forceinline__ F2 exp_pair(F2 x) {
  float a, b;
  mul2(x, F2(1.44269504f, 1.44269504f)).get(a, b);
  asm("ex2.approx.ftz.f32 %0, %0;\n" : "+f"(a));
  asm("ex2.approx.ftz.f32 %0, %0;\n" : "+f"(b));
  return F2(a, b);
}

// four codes of two pairs, packed: the rule of q8 (fp32 product, clamp, half away from zero)
template <bool Q127>
__device__ __forceinline__ uint32_t codes4(F2 x01, F2 x23, F2 inv, float qmax) {
  float y[4], h[4];
  mul2(x01, inv).get(y[0], y[1]);
  mul2(x23, inv).get(y[2], y[3]);
  int c[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    y[i] = fmaxf(y[i], Q127 ? -127.f : -qmax);  // at 127 the upper clamp is the saturating pack
    if (!Q127) y[i] = fminf(y[i], qmax);
    h[i] = copysignf(0.5f, y[i]);
  }
  add2(F2(y[0], y[1]), F2(h[0], h[1])).get(y[0], y[1]);
  add2(F2(y[2], y[3]), F2(h[2], h[3])).get(y[2], y[3]);
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] = __float2int_rz(y[i]);
  return pack_sat_s8x2(c[1], c[0], pack_sat_s8x2(c[3], c[2], 0u));
}
// the codes of a pair (the rule of q8) as fp32 values
__device__ __forceinline__ F2 code_pair(F2 x, float inv, float qmax) {
  float y0, y1;
  mul2(x, F2(inv, inv)).get(y0, y1);
  y0 = fminf(fmaxf(y0, -qmax), qmax);
  y1 = fminf(fmaxf(y1, -qmax), qmax);
  add2(F2(y0, y1), F2(copysignf(0.5f, y0), copysignf(0.5f, y1))).get(y0, y1);
  return F2(truncf(y0), truncf(y1));
}
// INT8 products accumulate on top of the bit pattern of 1.5 * 2^23 (|sum| <= 128 * 127 * 127 < 2^22): the accumulator read as
// a float is 1.5 * 2^23 + sum, and one subtraction gives the sum exactly, two at a time
__device__ __forceinline__ void mma_s8_biased(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0x4B400000));
}
__device__ __forceinline__ F2 unbias2(int a, int b) { return add2(F2(__int_as_float(a), __int_as_float(b)), F2(-12582912.f, -12582912.f)); }

// two fp32 values as three bf16 pairs, biggest first (8 + 8 + 8 bits: the sum is exact)
__device__ __forceinline__ void split3_pair(F2 x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  float a, b;
  x.get(a, b);
  hi = Act<__nv_bfloat16>::pack2(a, b);
  const F2 r = sub2(x, F2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)));
  r.get(a, b);
  mid = Act<__nv_bfloat16>::pack2(a, b);
  sub2(r, F2(__uint_as_float(mid << 16), __uint_as_float(mid & 0xffff0000u))).get(a, b);
  lo = Act<__nv_bfloat16>::pack2(a, b);
}
__device__ __forceinline__ void split3(const float (&x)[8], uint32_t (&hi)[4], uint32_t (&mid)[4], uint32_t (&lo)[4]) {
#pragma unroll
  for (int p = 0; p < 4; ++p) split3_pair(F2(x[2 * p], x[2 * p + 1]), hi[p], mid[p], lo[p]);
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

}  // namespace lq
