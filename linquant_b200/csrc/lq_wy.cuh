// WY-representation helpers shared by the delta-rule prologues: the blocked unit-lower-triangular inverse (forward substitution
// inside 16 x 16 blocks, the blocks below by doubling as 3xTF32 products) and the T . diag(cw) . B product with the left
// factor split into three bf16 pieces.
#pragma once
#include <type_traits>

#include "lq_common.cuh"

namespace lq {

__device__ __forceinline__ uint32_t tf32_rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float pow_exact01(float x, float e) { return e == 0.f ? 1.f : (e == 1.f ? x : powf(x, e)); }

// One warp: acc (an m16n8 fragment) += A . B[:, 8 nt ..] for 16 x 16 fp32 blocks in shared memory (row stride 68),
// both factors split into a TF32 part and a TF32 remainder (three MMAs per k-step; products good to about 2^-21).
__device__ __forceinline__ void blk16_mma(float (&acc)[4], const float* A, const float* B, int nt, int g, int j) {
#pragma unroll
  for (int kk = 0; kk < 2; ++kk) {
    const int c0 = 8 * kk + j, c1 = c0 + 4;
    const float xa[4] = {A[g * 68 + c0], A[(g + 8) * 68 + c0], A[g * 68 + c1], A[(g + 8) * 68 + c1]};
    uint32_t ab[4], as_[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      ab[e] = tf32_rna(xa[e]);
      as_[e] = tf32_rna(xa[e] - __uint_as_float(ab[e]));
    }
    const float y0 = B[c0 * 68 + 8 * nt + g], y1 = B[c1 * 68 + 8 * nt + g];
    const uint32_t b0 = tf32_rna(y0), b1 = tf32_rna(y1);
    const uint32_t s0 = tf32_rna(y0 - __uint_as_float(b0)), s1 = tf32_rna(y1 - __uint_as_float(b1));
    mma_tf32(acc, as_[0], as_[1], as_[2], as_[3], b0, b1);
    mma_tf32(acc, ab[0], ab[1], ab[2], ab[3], s0, s1);
    mma_tf32(acc, ab[0], ab[1], ab[2], ab[3], b0, b1);
  }
}
__device__ __forceinline__ void blk16_store(float* D, const float (&acc)[4], float sign, int nt, int g, int j) {
  *reinterpret_cast<float2*>(D + g * 68 + 8 * nt + 2 * j) = make_float2(sign * acc[0], sign * acc[1]);
  *reinterpret_cast<float2*>(D + (g + 8) * 68 + 8 * nt + 2 * j) = make_float2(sign * acc[2], sign * acc[3]);
}

// T = (I + G)^-1 for a strictly lower-triangular 64x64 G (both [64][68] fp32 in shared memory), 256 threads, as a
// blocked inverse over 16 x 16 blocks (reference: torch.linalg.solve_triangular, zoo/gated_delta_rule.py:40-41):
//   * the four diagonal blocks D_I = (I + G_II)^-1 by forward substitution, all at once: one column per group of four
//     lanes, sixteen steps, right-looking (lane r keeps the running sums of rows 4m + r; one shuffle per step), the
//     lane's elements of G read up front;
//   * by doubling, T_10 = -D_1 (G_10 D_0) and T_32 = -D_3 (G_32 D_2), then the 32 x 32 block below them, T_lo =
//     -[T of rows 32 ..] (G_lo [T of rows 0 .. 31]), as 16 x 8 tiles on the tensor cores (3xTF32), one warp a tile; the inner
//     products are parked in the unused upper blocks of T.
// A serial chain, bound by its latency: four dependent product stages (block column by block column there were six, of up to
// three products with two tiles each). Ends with every thread past a barrier.
__device__ __forceinline__ void wy_solve(const float* s_G, float* s_T) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, j = lane & 3;
  auto blkG = [&](int I, int J) { return s_G + (16 * I) * 68 + 16 * J; };
  auto blkT = [&](int I, int J) { return s_T + (16 * I) * 68 + 16 * J; };
  {  // diagonal blocks
    const int col = tid >> 2, r = tid & 3;  // global column; block I = col / 16
    const int I = col >> 4, cl = col & 15;
    const float* G = blkG(I, I);
    float* T = blkT(I, I);
    float4 gr[4][4];  // row 4m + r, columns 4n ..
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n <= m; ++n) gr[m][n] = *reinterpret_cast<const float4*>(G + (4 * m + r) * 68 + 4 * n);
    float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float val = (i == cl ? 1.f : 0.f) - part[i >> 2];
      val = __shfl_sync(0xffffffffu, val, (lane & ~3) | (i & 3));
      if (r == 0) T[i * 68 + cl] = val;
#pragma unroll
      for (int m = i >> 2; m < 4; ++m) {
        const float4 q = gr[m][i >> 2];
        const float gv = (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
        if (m > (i >> 2) || r > (i & 3)) part[m] = fmaf(gv, val, part[m]);
      }
    }
  }
  __syncthreads();
  const int nt = warp & 1, pr = warp >> 1;
  const int I1 = 2 * pr + 1;                // pairs of the first level: (1, 0) and (3, 2)
  const int I2 = 2 + (pr >> 1), J2 = pr & 1;  // blocks of the second
  if (pr < 2) {
    float acc[4] = {};
    blk16_mma(acc, blkG(I1, I1 - 1), blkT(I1 - 1, I1 - 1), nt, g, j);
    blk16_store(blkT(I1 - 1, I1), acc, 1.f, nt, g, j);
  }
  __syncthreads();
  if (pr < 2) {
    float acc[4] = {};
    blk16_mma(acc, blkT(I1, I1), blkT(I1 - 1, I1), nt, g, j);
    blk16_store(blkT(I1, I1 - 1), acc, -1.f, nt, g, j);
  }
  __syncthreads();
  {  // P = G_lo [D_0 0; T_10 D_1], parked in the transposed place
    float acc[4] = {};
    if (J2 == 0) blk16_mma(acc, blkG(I2, 0), blkT(0, 0), nt, g, j);
    blk16_mma(acc, blkG(I2, 1), blkT(1, J2), nt, g, j);
    blk16_store(blkT(J2, I2), acc, 1.f, nt, g, j);
  }
  __syncthreads();
  {  // T_lo = -[D_2 0; T_32 D_3] P
    float acc[4] = {};
    blk16_mma(acc, blkT(I2, 2), blkT(J2, 2), nt, g, j);
    if (I2 == 3) blk16_mma(acc, blkT(3, 3), blkT(J2, 3), nt, g, j);
    blk16_store(blkT(I2, J2), acc, -1.f, nt, g, j);
  }
  __syncthreads();
}

// ---- W = T diag(cw) B and U = T diag(cw) B on the tensor cores, eight warps, each a slice of the columns (tokens x columns B).
// T diag(cw) is split into three bf16 pieces (8 + 8 + 8 bits: exact) once, in the order of the MMA fragments; B comes in as
// one piece (bf16 values), two (fp16 values) or three (fp32 values). Products of two pieces are exact in fp32; they are
// accumulated smallest first. Rows g and g + 8 of an MMA are tokens 2g and 2g + 1 of the 16-token tile, so that a lane holds
// neighbouring tokens. Only the ten 16 x 16 tiles on and below the diagonal are kept: tile (mt, ks) at mt (mt + 1) / 2 + ks.

// fragments [10 tiles][3 pieces][32 lanes] of T diag(cw); T is [64][68] fp32
__device__ __forceinline__ void wy_fragments(const float* s_T, const float* s_cw, uint4* s_frag, int warp, int lane) {
  const int g = lane >> 2, j = lane & 3;
  for (int u = warp; u < 10; u += 8) {
    const int mt = u < 1 ? 0 : u < 3 ? 1 : u < 6 ? 2 : 3, ks = u - mt * (mt + 1) / 2;
    uint32_t p[3][4];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int col = 16 * ks + 8 * s + 2 * j;
      const float2 cw = *reinterpret_cast<const float2*>(s_cw + col);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 t = *reinterpret_cast<const float2*>(s_T + (16 * mt + 2 * g + r) * 68 + col);
        split3_pair(mul2(F2(t.x, t.y), F2(cw.x, cw.y)), p[0][2 * s + r], p[1][2 * s + r], p[2][2 * s + r]);
      }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) s_frag[(3 * u + i) * 32 + lane] = make_uint4(p[i][0], p[i][1], p[i][2], p[i][3]);
  }
}

// The same for two factors; T lies in the second half of the fragments' place: all of it is read before any is written.
__device__ __forceinline__ void wy_fragments2(const float* s_T, const float* s_cw0, const float* s_cw1, uint4* s_frag, int warp, int lane) {
  const int g = lane >> 2, j = lane & 3;
  float2 t[2][4];
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int u = warp + 8 * it;
    if (u < 10) {
      const int mt = u < 1 ? 0 : u < 3 ? 1 : u < 6 ? 2 : 3, ks = u - mt * (mt + 1) / 2;
#pragma unroll
      for (int i = 0; i < 4; ++i) t[it][i] = *reinterpret_cast<const float2*>(s_T + (16 * mt + 2 * g + (i & 1)) * 68 + 16 * ks + 8 * (i >> 1) + 2 * j);
    }
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int u = warp + 8 * it;
    if (u < 10) {
      const int mt = u < 1 ? 0 : u < 3 ? 1 : u < 6 ? 2 : 3, ks = u - mt * (mt + 1) / 2;
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const float* s_cw = f ? s_cw1 : s_cw0;
        uint32_t p[3][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 cw = *reinterpret_cast<const float2*>(s_cw + 16 * ks + 8 * (i >> 1) + 2 * j);
          split3_pair(mul2(F2(t[it][i].x, t[it][i].y), F2(cw.x, cw.y)), p[0][i], p[1][i], p[2][i]);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) s_frag[(30 * f + 3 * u + i) * 32 + lane] = make_uint4(p[i][0], p[i][1], p[i][2], p[i][3]);
      }
    }
  }
}

// B fragments (16 tokens x 8 NT columns) of 16-bit rows in shared memory: raw[nt][s] = tokens 8 s + 2 j, + 1 of column 8 nt + g
template <int NT, typename T>
__device__ __forceinline__ void wy_ldmatrix(uint32_t (&raw)[NT][2], const T* s, int ld, int lane) {
  const uint32_t p = (uint32_t)__cvta_generic_to_shared(s + (lane & 15) * ld + (NT == 2 ? 8 * (lane >> 4) : 0));
  if constexpr (NT == 2)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(raw[0][0]), "=r"(raw[0][1]), "=r"(raw[1][0]), "=r"(raw[1][1]) : "r"(p) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(raw[0][0]), "=r"(raw[0][1]) : "r"(p) : "memory");
}

// acc[mt][nt] = rows 16 mt .. of T diag(cw) B; operand(ks, pieces) delivers the NB pieces of the B fragments of tokens 16 ks ..
template <int NT, int NB, typename F>
__device__ __forceinline__ void wy_product3(float (&acc)[4][NT][4], const uint4* s_frag, int lane, F operand) {
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = acc[mt][nt][2] = acc[mt][nt][3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    uint32_t b[NB][NT][2];
    operand(ks, b);
#pragma unroll
    for (int mt = ks; mt < 4; ++mt) {
      const uint4* f = s_frag + 3 * (mt * (mt + 1) / 2 + ks) * 32 + lane;
      const uint4 hi = f[0], mid = f[32], lo = f[64];
      auto mma = [&](const uint4& x, int i) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_bf16(acc[mt][nt], x.x, x.y, x.z, x.w, b[i][nt][0], b[i][nt][1]);
      };
      if (NB == 2) mma(lo, NB - 1);
      mma(lo, 0);
      if (NB == 3) mma(hi, NB - 1);
      if (NB >= 2) mma(mid, NB >= 2 ? 1 : 0);
      mma(mid, 0);
      if (NB >= 2) mma(hi, NB >= 2 ? 1 : 0);
      mma(hi, 0);
    }
  }
}

// bf16 or fp16 rows of shared memory as the B operand: one exact piece, or two
template <typename T, int NT>
__device__ __forceinline__ void wy_pieces16(uint32_t (&b)[std::is_same<T, __half>::value ? 2 : 1][NT][2], const T* s, int ld, int lane) {
  wy_ldmatrix<NT>(b[0], s, ld, lane);
  if constexpr (std::is_same<T, __half>::value) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int s2 = 0; s2 < 2; ++s2) {
        const float x0 = Act<T>::get(b[0][nt][s2], 0), x1 = Act<T>::get(b[0][nt][s2], 1);
        const uint32_t hi = Act<__nv_bfloat16>::pack2(x0, x1);
        b[0][nt][s2] = hi;
        b[1][nt][s2] = Act<__nv_bfloat16>::pack2(x0 - __uint_as_float(hi << 16), x1 - __uint_as_float(hi & 0xffff0000u));
      }
  }
}

// codes of W, columns n0 .. n0 + 8 NT: a lane pair (j even, odd) exchanges so that the even one stores four channels of token
// 2g and the odd one those of token 2g + 1
template <typename T, int NT>
__device__ __forceinline__ void wy_store_w(const float (&acc)[4][NT][4], int8_t* wq, int n0, float inv_sw, float qmax, int lane) {
  const int g = lane >> 2, j = lane & 3, odd = j & 1;
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const uint32_t r0 = Act<T>::pack2(acc[mt][nt][0], acc[mt][nt][1]), r1 = Act<T>::pack2(acc[mt][nt][2], acc[mt][nt][3]);
      const uint32_t w = codes4<false>(F2(Act<T>::get(r0, 0), Act<T>::get(r0, 1)), F2(Act<T>::get(r1, 0), Act<T>::get(r1, 1)), F2(inv_sw, inv_sw), qmax);
      const uint32_t other = __shfl_xor_sync(0xffffffffu, w, 1);  // low half: token 2g, high half: 2g + 1
      const uint32_t word = odd ? __byte_perm(other, w, 0x7632) : __byte_perm(w, other, 0x5410);
      *reinterpret_cast<uint32_t*>(wq + wq_offset(16 * mt + 2 * g + odd, n0 + 8 * nt + 4 * (j >> 1))) = word;
    }
}

// U = T diag(cw) v for all V columns, stored [V][64] in the activation dtype
template <typename T, int V>
__device__ __forceinline__ void wy_u(const uint4* s_frag, const T* s_v, int ldv, T* u, int warp, int lane) {
  constexpr int NT = V / 64, NB = std::is_same<T, __half>::value ? 2 : 1;
  const int n0 = (V / 8) * warp, g = lane >> 2, j = lane & 3;
  float acc[4][NT][4];
  wy_product3<NT, NB>(acc, s_frag, lane, [&](int ks, uint32_t (&b)[NB][NT][2]) { wy_pieces16<T, NT>(b, s_v + 16 * ks * ldv + n0, ldv, lane); });
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        *reinterpret_cast<uint32_t*>(u + (size_t)(n0 + 8 * nt + 2 * j + e) * 64 + 16 * mt + 2 * g) = Act<T>::pack2(acc[mt][nt][e], acc[mt][nt][2 + e]);
}

}  // namespace lq
