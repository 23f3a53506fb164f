// Diagonal (per-channel) decay cells: GLA (linear family) and KDA (delta family).
//
// Three chunk-parallel kernels, one CTA per (batch*head, chunk):
//   rows   chunk-local cumulative log-decay per channel (double accumulate), log envelope, pre-decayed q_read codes,
//          gated k_write codes (Omega * s^-eta), and for the linear family the v_local / v_write codes
//   amat   the intra-chunk matrix A in 16-token secondary chunks: off-diagonal blocks as INT8 MMAs on operands
//          re-scaled around the block's anchor row (optionally rotated by a signed Hadamard on fp16-rounded values),
//          diagonal blocks as an fp32 reduction with the exact per-channel weights on the dequantised codes
//   kda_wy KDA only: unquantised Gram matrix with per-channel weights, (I+G)^-1, W codes, U
// The state pass and the output kernel are the scalar-decay kernels instantiated with per-channel carry decay
// and a precomputed A.
//
// Reference arithmetic: zoo/gla.py:27-63 (_gla_A_inter), :66-99 (_gla_A_intra), :103-148 (state), :171-213 (output),
// :249-250 (cumsum, envelope); zoo/kda.py:22-53 (_prep); reference.py:125-152, :155-163.
#include "lq_wy.cuh"
#include "lq_zoo_rows.cuh"

namespace lq {

struct DiagArgs {
  const void *q, *k, *v;
  const float *g, *beta, *signs;
  const float *sq, *sk, *skw, *svl, *svw, *sw;
  int8_t *qq, *kwT, *vlT, *vwT, *wq;
  float *gc, *genv, *gcl, *fw;
  void* u;
  __half* amat;
  int T, H, NT;
  float scale, eta, sigma, tau, qmax;
};

template <int K, int BATCH = 64 * K / 4 / 256>
__device__ __forceinline__ void load_gc_tile(const float* gc_tile, float* s_gc) {  // 256 threads
  // BATCH 16-byte loads of the thread are requested before the first of them is stored (one or two trips to memory
  // instead of one per load)
  constexpr int NIT = 64 * K / 4 / 256;
#pragma unroll
  for (int b0 = 0; b0 < NIT; b0 += BATCH) {
    float4 v[BATCH];
#pragma unroll
    for (int it = 0; it < BATCH; ++it) v[it] = __ldg(reinterpret_cast<const float4*>(gc_tile) + threadIdx.x + 256 * (b0 + it));
#pragma unroll
    for (int it = 0; it < BATCH; ++it) {
      const int i = threadIdx.x + 256 * (b0 + it), t = i / (K / 4), c4 = i % (K / 4);
      *reinterpret_cast<float4*>(s_gc + t * (K + 4) + 4 * c4) = v[it];
    }
  }
}

// ------------------------------------------------------------------------------------------------ rows
template <typename T, int K, int V, bool DELTA>
__global__ void __launch_bounds__(256) zoo_diag_rows_kernel(DiagArgs a) {
  pdl_enter();
  constexpr int C = 64, LD = K + 4;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* s_gc = reinterpret_cast<float*>(smem_raw);
  float* s_le = s_gc + C * LD;
  float* s_hw = s_le + C;
  uint32_t(*s_kw)[17] = reinterpret_cast<uint32_t(*)[17]>(s_hw + C);
  uint32_t(*s_vl)[17] = s_kw + K;
  uint32_t(*s_vw)[17] = s_vl + V;

  const int c = blockIdx.x, bh = blockIdx.y;
  const int b = bh / a.H, h = bh % a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t tile = (size_t)bh * a.NT + c;
  const float e_hw = (1.f - a.sigma) * a.tau;

  // stage the raw log-decays of the chunk (coalesced), then one thread per channel scans them in double
  {
    constexpr int NIT = C * (K / 4) / 256;
    float4 v[NIT];
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int i = tid + 256 * it, t = i / (K / 4), c4 = i % (K / 4);
      v[it] = __ldg(reinterpret_cast<const float4*>(a.g + (((size_t)b * a.T + (size_t)c * C + t) * a.H + h) * K) + c4);
    }
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int i = tid + 256 * it, t = i / (K / 4), c4 = i % (K / 4);
      *reinterpret_cast<float4*>(s_gc + t * LD + 4 * c4) = v[it];
    }
  }
  if (DELTA && tid >= 128 && tid < 128 + C) {
    const int t = tid - 128;
    const float bt = a.beta[((size_t)b * a.T + (size_t)c * C + t) * a.H + h];
    s_hw[t] = pow_exact01(bt, e_hw);
  }
  __syncthreads();
  if (tid < K) {
    double acc = 0.0;
    float f = 0.f;
#pragma unroll 8
    for (int t = 0; t < C; ++t) {
      acc += (double)s_gc[t * LD + tid];
      f = (float)acc;
      s_gc[t * LD + tid] = f;
    }
    a.gcl[tile * K + tid] = expf(f);
  }
  __syncthreads();
  for (int i = tid; i < C * (K / 4); i += 256) {
    const int t = i / (K / 4), c4 = i % (K / 4);
    reinterpret_cast<float4*>(a.gc + (tile * C + t) * K)[c4] = *reinterpret_cast<const float4*>(s_gc + t * LD + 4 * c4);
  }
  __syncthreads();
  for (int tt = 0; tt < 8; ++tt) {
    const int t = 8 * warp + tt;
    float m = -INFINITY;
    for (int n = lane; n < K; n += 32) m = fmaxf(m, s_gc[(C - 1) * LD + n] - s_gc[t * LD + n]);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    if (lane == 0) {
      s_le[t] = m;
      a.genv[tile * C + t] = expf(a.eta * m);
    }
  }
  __syncthreads();

  {
    constexpr int LPR = K / 8, G = 32 / LPR;
    const int r = lane % LPR, grp = lane / LPR;
    const float inv_sq = 1.0f / a.sq[h];
    float inv_kw[8], gl[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      inv_kw[j] = 1.0f / a.skw[h * K + 8 * r + j];
      gl[j] = s_gc[(C - 1) * LD + 8 * r + j];
    }
    const T* qp = reinterpret_cast<const T*>(a.q);
    const T* kp = reinterpret_cast<const T*>(a.k);
    for (int tg = warp * G + grp; tg < C / 4; tg += 8 * G) {
      uint32_t kwp[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) kwp[j] = 0u;
      // the eight row loads of the group are in flight before the first is used
      uint4 rq[4], rk[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const size_t row = (((size_t)b * a.T + (size_t)c * C + 4 * tg + i) * a.H + h) * K + 8 * r;
        rq[i] = __ldg(reinterpret_cast<const uint4*>(qp + row));
        rk[i] = __ldg(reinterpret_cast<const uint4*>(kp + row));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = 4 * tg + i;
        float x[8], gv[8];
        int cd[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) gv[j] = s_gc[t * LD + 8 * r + j];
        Act<T>::unpack8(rq[i], x);
#pragma unroll
        for (int j = 0; j < 8; ++j) cd[j] = q8(__fmul_rn(__fmul_rn(x[j], __expf(gv[j])), a.scale), inv_sq, a.qmax);
        *reinterpret_cast<uint2*>(a.qq + (tile * C + t) * K + 8 * r) =
            make_uint2(pack4(cd[0], cd[1], cd[2], cd[3]), pack4(cd[4], cd[5], cd[6], cd[7]));
        Act<T>::unpack8(rk[i], x);
        if (DELTA && e_hw != 0.f) {
          const float hw = s_hw[t];
#pragma unroll
          for (int j = 0; j < 8; ++j) x[j] = Act<T>::round(__fmul_rn(x[j], hw));
        }
        const float ele = a.eta * s_le[t];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float w = __expf(__fsub_rn(__fsub_rn(gl[j], gv[j]), ele));
          kwp[j] |= ((uint32_t)q8(__fmul_rn(x[j], w), inv_kw[j], a.qmax) & 0xffu) << (8 * i);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s_kw[8 * r + j][tg] = kwp[j];
    }
  }
  if (!DELTA) {
    constexpr int LPR = V / 8, G = 32 / LPR;
    const int r = lane % LPR, grp = lane / LPR;
    float inv_vl[8], inv_vw[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      inv_vl[j] = 1.0f / a.svl[h * V + 8 * r + j];
      inv_vw[j] = 1.0f / a.svw[h * V + 8 * r + j];
    }
    const T* vp = reinterpret_cast<const T*>(a.v);
    for (int tg = warp * G + grp; tg < C / 4; tg += 8 * G) {
      uint32_t vlp[8], vwp[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) vlp[j] = vwp[j] = 0u;
      uint4 rv[4];  // the four row loads of the group are in flight before the first is used
#pragma unroll
      for (int i = 0; i < 4; ++i)
        rv[i] = __ldg(reinterpret_cast<const uint4*>(vp + (((size_t)b * a.T + (size_t)c * C + 4 * tg + i) * a.H + h) * V + 8 * r));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = 4 * tg + i;
        float x[8];
        Act<T>::unpack8(rv[i], x);
        const float fv = expf(a.eta * s_le[t]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          vlp[j] |= ((uint32_t)q8(x[j], inv_vl[j], a.qmax) & 0xffu) << (8 * i);
          vwp[j] |= ((uint32_t)q8(__fmul_rn(x[j], fv), inv_vw[j], a.qmax) & 0xffu) << (8 * i);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s_vl[8 * r + j][tg] = vlp[j];
        s_vw[8 * r + j][tg] = vwp[j];
      }
    }
  }
  __syncthreads();
  uint32_t* kw_out = reinterpret_cast<uint32_t*>(a.kwT + tile * (size_t)(K * C));
  for (int i = tid; i < K * 16; i += 256) kw_out[i] = s_kw[i >> 4][i & 15];
  if (!DELTA) {
    uint32_t* vl_out = reinterpret_cast<uint32_t*>(a.vlT + tile * (size_t)(V * C));
    uint32_t* vw_out = reinterpret_cast<uint32_t*>(a.vwT + tile * (size_t)(V * C));
    for (int i = tid; i < V * 16; i += 256) {
      vl_out[i] = s_vl[i >> 4][i & 15];
      vw_out[i] = s_vw[i >> 4][i & 15];
    }
  }
}

// ------------------------------------------------------------------------------------------------ A matrix
// Eight warps, no data shared but the log-decay tile and the codes of the off-diagonal operands; every operand element is
// made in the register of the MMA fragment that contracts it. In all tiles a lane holds of its two rows (g, g + 8 of 16) the
// channels 32 m + 8 j .. + 7 (one 16-byte load each): the contraction index may be dealt to the MMA slots in any order as
// long as both operands agree.
//   warps 0 - 3   diagonal block I = warp: both operands' codes, times exp(g - a) and exp(a - g) around the block's first row
//                 a, each split into three bf16 pieces (exact), six products (big to small down to 2^-16) on the tensor cores
//   warps 4 - 7   the nine re-scaled operand tiles of the off-diagonal block rows: fp16 rounding, Hadamard rotation, codes; then
//                 (one barrier of these four warps) the six 16 x 16 INT8 products
// The 2^7 (2^6) Hadamard transform is split over the channel bits: bits 0, 1, 3, 4 are the sixteen slots of an m16n8k16 product
// with the +-1 matrix (exact operands, fp32 accumulation), the others a butterfly between a lane's own registers.
// Bound by instruction issue. The kernel before it (operands through shared memory, shuffle butterflies, 3xTF32 with the
// split in the product loop: 42 k warp instructions and 27 block barriers per chunk) took 2070 us for 256 (b, h) x 128 chunks at K = 128; this one 1637.
template <typename T, int K>
__global__ void __launch_bounds__(256) zoo_diag_amat_kernel(DiagArgs a) {
  pdl_enter();
  constexpr int C = 64, LD = K + 4, SUB = 16, M = K / 32;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* s_gc = reinterpret_cast<float*>(smem_raw);                          // [C][LD]
  float* s_sgn = s_gc + C * LD;                                              // [K] rotation signs / sqrt(K) on the fp16 grid
  float* s_hw = s_sgn + K;                                                   // [C]
  uint4* s_code = reinterpret_cast<uint4*>(s_hw + C);                        // [9 tiles][M][32 lanes]: row g (eh 0, 1), row g + 8

  const int c = blockIdx.x, bh = blockIdx.y;
  const int b = bh / a.H, h = bh % a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, j = lane & 3;
  const size_t tile = (size_t)bh * a.NT + c;
  const float e_hw = (1.f - a.sigma) * a.tau;
  const bool use_hw = a.beta != nullptr && e_hw != 0.f;
  const bool rot = a.signs != nullptr;
  const T* qp = reinterpret_cast<const T*>(a.q);
  const T* kp = reinterpret_cast<const T*>(a.k);
  auto grow = [&](int t) { return (((size_t)b * a.T + (size_t)c * C + t) * a.H + h) * K + 8 * j; };

  load_gc_tile<K, K / 32>(a.gc + tile * (size_t)(C * K), s_gc);
  if (tid < C) s_hw[tid] = use_hw ? pow_exact01(a.beta[((size_t)b * a.T + (size_t)c * C + tid) * a.H + h], e_hw) : 1.f;
  if (tid >= 128 && tid < 128 + K) {
    const float n16 = __half2float(__float2half_rn(K == 64 ? 0.125f : 0.08838834764831845f));
    s_sgn[tid - 128] = rot ? a.signs[tid - 128] * n16 : 1.f;
  }
  __syncthreads();

  const float fq = 1.0f / a.sq[h], fk = 1.0f / a.sk[h];
  const float sqk = __fmul_rn(a.sq[h], a.sk[h]);
  __half* A = a.amat + tile * (size_t)(C * C);
  auto lds8 = [&](const float* p, float (&v)[8]) {
    *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
    *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(p + 4);
  };

  if (warp < 4) {
    // ---------------------------------------------------------------------------------- diagonal block
    const int t0 = SUB * warp;
    uint4 rq[2][M], rk[2][M];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) {
        rq[r][m] = __ldg(reinterpret_cast<const uint4*>(qp + grow(t0 + g + 8 * r) + 32 * m));
        rk[r][m] = __ldg(reinterpret_cast<const uint4*>(kp + grow(t0 + g + 8 * r) + 32 * m));
      }
    auto key = [&](const uint4& raw, int t, float (&x)[8]) {  // the readout key of one row piece
      Act<T>::unpack8(raw, x);
      if (use_hw) {
        const float hw = s_hw[t];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = Act<T>::round(__fmul_rn(x[e], hw));
      }
    };
    // the weight exp(g_i - g_j) factors around the first row unless the decay across the block is so strong (beyond e^60) that
    // the second factor could leave fp32
    float spread = 0.f;
    for (int n = lane; n < K; n += 32) spread = fmaxf(spread, __fsub_rn(s_gc[t0 * LD + n], s_gc[(t0 + SUB - 1) * LD + n]));
    const bool exact = __any_sync(0xffffffffu, spread > 60.f);
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    if (!exact) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float an[8];
        lds8(s_gc + t0 * LD + 32 * m + 8 * j, an);
        uint32_t qh[2][4], qm[2][4], ql[2][4], kh[2][4], km[2][4], kl[2][4];  // [row half][pair of channels]
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int t = t0 + g + 8 * r;
          float x[8], gv[8], e1[8];
          lds8(s_gc + t * LD + 32 * m + 8 * j, gv);
          Act<T>::unpack8(rq[r][m], x);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            e1[e] = __fsub_rn(gv[e], an[e]);
            x[e] = __fmul_rn((float)q8(__fmul_rn(x[e], a.scale), fq, a.qmax), __expf(e1[e]));
          }
          split3(x, qh[r], qm[r], ql[r]);
          key(rk[r][m], t, x);
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = __fmul_rn((float)q8(x[e], fk, a.qmax), __expf(-e1[e]));
          split3(x, kh[r], km[r], kl[r]);
        }
#pragma unroll
        for (int eh = 0; eh < 2; ++eh) {
          const int p = 2 * eh;
          auto mma = [&](float (&d)[4], const uint32_t (&qa)[2][4], const uint32_t (&kb)[4]) {
            mma_bf16(d, qa[0][p], qa[1][p], qa[0][p + 1], qa[1][p + 1], kb[p], kb[p + 1]);
          };
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            mma(acc[nt], ql, kh[nt]);
            mma(acc[nt], qh, kl[nt]);
            mma(acc[nt], qm, km[nt]);
            mma(acc[nt], qm, kh[nt]);
            mma(acc[nt], qh, km[nt]);
            mma(acc[nt], qh, kh[nt]);
          }
        }
      }
    } else {
      // one exp per (i, j, channel), a lane for each of its eight (i, j) of the accumulator layout
      for (int n = 0; n < K; ++n) {
        float qc[2], kc[2][2], gi[2], gj[2][2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int t = t0 + g + 8 * r;
          gi[r] = s_gc[t * LD + n];
          qc[r] = (float)q8(__fmul_rn(Act<T>::to(qp[grow(t) - 8 * j + n]), a.scale), fq, a.qmax);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int tj = t0 + 8 * r + 2 * j + e;
            gj[r][e] = s_gc[tj * LD + n];
            float x = Act<T>::to(kp[grow(tj) - 8 * j + n]);
            if (use_hw) x = Act<T>::round(__fmul_rn(x, s_hw[tj]));
            kc[r][e] = (float)q8(x, fk, a.qmax);
          }
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            acc[nt][i] = fmaf(__fmul_rn(qc[i >> 1], kc[nt][i & 1]), __expf(gi[i >> 1] - gj[nt][i & 1]), acc[nt][i]);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = g + 8 * r, jj = 8 * nt + 2 * j;
        const float x0 = jj <= i ? __fmul_rn(acc[nt][2 * r], sqk) : 0.f, x1 = jj + 1 <= i ? __fmul_rn(acc[nt][2 * r + 1], sqk) : 0.f;
        *reinterpret_cast<uint32_t*>(A + (t0 + i) * C + t0 + jj) = Act<__half>::pack2(x0, x1);
      }
    return;
  }

  // ------------------------------------------------------------------------------------ off-diagonal operand tiles
  // tile I - 1: the sixteen query rows of block row I; tiles 3 + (I - 1) I / 2 + J: key rows of block J, both around row 16 I
  const int w4 = warp - 4;
  const uint32_t had = [&]() {  // (-1)^popc(s & n) for slots s = 2j, 2j + 1 and column n = g, as two halves
    const uint32_t s0 = (__popc((2 * j) & g) & 1) ? 0xBC00u : 0x3C00u, s1 = (__popc((2 * j + 1) & g) & 1) ? 0xBC00u : 0x3C00u;
    return s0 | (s1 << 16);
  }();
  const bool q127 = a.qmax == 127.f;
  for (int it = w4; it < 9; it += 4) {
    const bool isq = it < 3;
    const int u = it - 3;
    const int I = isq ? it + 1 : (u < 1 ? 1 : u < 3 ? 2 : 3);
    const int t0 = SUB * (isq ? I : u - (I - 1) * I / 2);
    const T* src = isq ? qp : kp;
    uint4 raw[2][M];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m) raw[r][m] = __ldg(reinterpret_cast<const uint4*>(src + grow(t0 + g + 8 * r) + 32 * m));
    F2 y[M][2][2][2];  // [m][eh][row half][channel pair]
#pragma unroll
    for (int m = 0; m < M; ++m) {
      float an[8], x[2][8];
      lds8(s_gc + SUB * I * LD + 32 * m + 8 * j, an);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int t = t0 + g + 8 * r;
        float gv[8];
        lds8(s_gc + t * LD + 32 * m + 8 * j, gv);
        Act<T>::unpack8(raw[r][m], x[r]);
        if (isq) {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[r][e] = __fmul_rn(__fmul_rn(x[r][e], __expf(__fsub_rn(gv[e], an[e]))), a.scale);
        } else {
          if (use_hw) {
            const float hw = s_hw[t];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[r][e] = Act<T>::round(__fmul_rn(x[r][e], hw));
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) x[r][e] = __fmul_rn(x[r][e], __expf(__fsub_rn(an[e], gv[e])));
        }
      }
#pragma unroll
      for (int eh = 0; eh < 2; ++eh) {
        if (rot) {
          uint32_t f[2][2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            f[r][0] = Act<__half>::pack2(x[r][4 * eh], x[r][4 * eh + 1]);
            f[r][1] = Act<__half>::pack2(x[r][4 * eh + 2], x[r][4 * eh + 3]);
          }
          float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
          mma_f16(d0, f[0][0], f[1][0], f[0][1], f[1][1], had, had);
          mma_f16(d1, f[0][0], f[1][0], f[0][1], f[1][1], had, had ^ 0x80008000u);
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            y[m][eh][r][0] = F2(d0[2 * r], d0[2 * r + 1]);
            y[m][eh][r][1] = F2(d1[2 * r], d1[2 * r + 1]);
          }
        } else {
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            y[m][eh][r][0] = F2(x[r][4 * eh], x[r][4 * eh + 1]);
            y[m][eh][r][1] = F2(x[r][4 * eh + 2], x[r][4 * eh + 3]);
          }
        }
      }
    }
    if (rot) {  // the remaining channel bits: 2 (eh), 5 and 6 (m)
      const F2 neg(-1.f, -1.f);
      auto fly = [&](F2& p, F2& q) {
        const F2 s = add2(p, q);
        q = fma2(q, neg, p);
        p = s;
      };
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
          for (int m = 0; m < M; ++m) fly(y[m][0][r][e], y[m][1][r][e]);
#pragma unroll
          for (int eh = 0; eh < 2; ++eh) {
#pragma unroll
            for (int m = 0; m < M; m += 2) fly(y[m][eh][r][e], y[m + 1][eh][r][e]);
            if (M == 4) {
              fly(y[0][eh][r][e], y[2 % M][eh][r][e]);
              fly(y[1][eh][r][e], y[3 % M][eh][r][e]);
            }
          }
        }
    }
    const float inv1 = isq ? fq : fk;
    const F2 inv(inv1, inv1);
#pragma unroll
    for (int m = 0; m < M; ++m) {
      uint32_t w[2][2];
#pragma unroll
      for (int eh = 0; eh < 2; ++eh) {
        const float4 sg = *reinterpret_cast<const float4*>(s_sgn + 32 * m + 8 * j + 4 * eh);
        const F2 s0(sg.x, sg.y), s1(sg.z, sg.w);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const F2 y0 = rot ? mul2(y[m][eh][r][0], s0) : y[m][eh][r][0], y1 = rot ? mul2(y[m][eh][r][1], s1) : y[m][eh][r][1];
          w[r][eh] = q127 ? codes4<true>(y0, y1, inv, 127.f) : codes4<false>(y0, y1, inv, a.qmax);
        }
      }
      s_code[(it * M + m) * 32 + lane] = make_uint4(w[0][0], w[1][0], w[0][1], w[1][1]);
    }
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  for (int u = w4; u < 6; u += 4) {  // block (I, J)
    const int I = u < 1 ? 1 : u < 3 ? 2 : 3, J = u - (I - 1) * I / 2;
    int acc[2][4];
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const uint4 qa = s_code[((I - 1) * M + m) * 32 + lane], kb = s_code[((3 + u) * M + m) * 32 + lane];
      if (m == 0) {
        mma_s8_first(acc[0], qa.x, qa.y, qa.z, qa.w, kb.x, kb.z);
        mma_s8_first(acc[1], qa.x, qa.y, qa.z, qa.w, kb.y, kb.w);
      } else {
        mma_s8(acc[0], qa.x, qa.y, qa.z, qa.w, kb.x, kb.z);
        mma_s8(acc[1], qa.x, qa.y, qa.z, qa.w, kb.y, kb.w);
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = g + 8 * r, jj = 8 * nt + 2 * j;
        *reinterpret_cast<uint32_t*>(A + (SUB * I + i) * C + SUB * J + jj) =
            Act<__half>::pack2(__fmul_rn((float)acc[nt][2 * r], sqk), __fmul_rn((float)acc[nt][2 * r + 1], sqk));
        *reinterpret_cast<uint32_t*>(A + (SUB * J + i) * C + SUB * I + jj) = 0u;  // the block above the diagonal
      }
  }
}

// ------------------------------------------------------------------------------------------------ KDA WY prep
// Gram matrix G[i][j] = beta_i^sigma beta_j^(1-sigma) sum_n k[i,n] k[j,n] exp(gc[i,n] - gc[j,n]), i > j, in 16-token
// secondary chunks like the A matrix: inside a diagonal block every (i, j, n) takes its own exp (exponent <= 0);
// for block row I against the earlier tokens the operands are re-scaled around the anchor row 16 I,
//   kd[i,n] = k[i,n] exp(gc[i,n] - gc[16I,n]),  ke[j,n] = k[j,n] exp(gc[16I,n] - gc[j,n])   (both factors <= 1),
// and contracted on the tensor cores as 3xTF32 (big*big + big*small + small*big), which keeps fp32-grade products.
// W and U are T diag(beta^sigma) times k exp(gc) (3xTF32, both operands split) and times v (exact in TF32).
template <typename T, int K>
__device__ __forceinline__ void kda_scaled_rows(const DiagArgs& a, int b, int c, int h, const float* s_gc, float* s_x,
                                                int anchor_row, int first_row, int nrows, int dst_row, bool toward_anchor) {
  // rows [first_row, first_row + nrows) of k, times exp(gc[row] - gc[anchor]) (toward_anchor) or exp(gc[anchor] - gc[row]),
  // or times exp(gc[row]) when anchor_row < 0; written as fp32 to s_x rows dst_row ...
  constexpr int C = 64, LD = K + 4, LPR = K / 8, MAXIT = C * LPR / 256;
  const T* kp = reinterpret_cast<const T*>(a.k);
  // every row piece of the thread is requested before the first is used (at most MAXIT of them: nrows <= 64)
  uint4 raw[MAXIT];
#pragma unroll
  for (int it = 0; it < MAXIT; ++it) {
    const int i = threadIdx.x + 256 * it;
    if (i < nrows * LPR) {
      const int rr = i / LPR, seg = i % LPR;
      raw[it] = __ldg(reinterpret_cast<const uint4*>(kp + (((size_t)b * a.T + (size_t)c * C + first_row + rr) * a.H + h) * K + 8 * seg));
    }
  }
#pragma unroll
  for (int it = 0; it < MAXIT; ++it) {
    const int i = threadIdx.x + 256 * it;
    if (i >= nrows * LPR) break;
    const int rr = i / LPR, seg = i % LPR;
    const int t = first_row + rr;
    float x[8];
    Act<T>::unpack8(raw[it], x);
    const float4 g0 = *reinterpret_cast<const float4*>(s_gc + t * LD + 8 * seg);
    const float4 g1 = *reinterpret_cast<const float4*>(s_gc + t * LD + 8 * seg + 4);
    float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
    if (anchor_row >= 0) {
      const float4 a0 = *reinterpret_cast<const float4*>(s_gc + anchor_row * LD + 8 * seg);
      const float4 a1 = *reinterpret_cast<const float4*>(s_gc + anchor_row * LD + 8 * seg + 4);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) gv[e] = toward_anchor ? __fsub_rn(gv[e], av[e]) : __fsub_rn(av[e], gv[e]);
    }
    float y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = __fmul_rn(x[e], __expf(gv[e]));
    *reinterpret_cast<float4*>(s_x + (dst_row + rr) * LD + 8 * seg) = make_float4(y[0], y[1], y[2], y[3]);
    *reinterpret_cast<float4*>(s_x + (dst_row + rr) * LD + 8 * seg + 4) = make_float4(y[4], y[5], y[6], y[7]);
  }
}

template <typename T, int K, int V>
__global__ void __launch_bounds__(256) zoo_kda_wy_kernel(DiagArgs a) {
  pdl_enter();
  constexpr int C = 64, LD = K + 4, LDV = V + 8, SUB = 16;
  constexpr int REG0 = C * (LD > LDV ? LD : LDV);
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* s_gc = reinterpret_cast<float*>(smem_raw);  // gc tile; v (fp32) once the decayed keys are formed
  float* s_x = s_gc + REG0;                          // k (fp32), then anchored operands, then k exp(gc)
  float* s_G = s_x + C * LD;
  float* s_T = s_G + C * 68;
  float* s_bs = s_T + C * 68;
  float* s_b1 = s_bs + C;
  float* s_part = s_b1 + C;  // [8 warps][16][16] partial diagonal blocks
  float* s_vf = s_gc;

  const int c = blockIdx.x, bh = blockIdx.y;
  const int b = bh / a.H, h = bh % a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, j4 = lane & 3;
  const size_t tile = (size_t)bh * a.NT + c;

  load_gc_tile<K>(a.gc + tile * (size_t)(C * K), s_gc);
  {
    const T* kp = reinterpret_cast<const T*>(a.k);
    constexpr int NIT = C * (K / 8) / 256;
    uint4 raw[NIT];
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int i = tid + 256 * it, t = i / (K / 8), seg = i % (K / 8);
      raw[it] = __ldg(reinterpret_cast<const uint4*>(kp + (((size_t)b * a.T + (size_t)c * C + t) * a.H + h) * K + 8 * seg));
    }
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int i = tid + 256 * it, t = i / (K / 8), seg = i % (K / 8);
      float x[8];
      Act<T>::unpack8(raw[it], x);
      *reinterpret_cast<float4*>(s_x + t * LD + 8 * seg) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(s_x + t * LD + 8 * seg + 4) = make_float4(x[4], x[5], x[6], x[7]);
    }
  }
  if (tid < C) {
    const float bt = a.beta[((size_t)b * a.T + (size_t)c * C + tid) * a.H + h];
    s_bs[tid] = pow_exact01(bt, a.sigma);
    s_b1[tid] = pow_exact01(bt, 1.f - a.sigma);
    a.fw[tile * C + tid] = pow_exact01(bt, (1.f - a.sigma) * (1.f - a.tau));
  }
  for (int i = tid; i < C * 68; i += 256) s_G[i] = 0.f;
  __syncthreads();

  // ---- diagonal blocks (strictly lower pairs of each 16 x 16 block). As in the A matrix the per-channel weight
  // exp(gc_in - gc_jn) factors around the block's first row a into exp(gc_in - a_n) (<= 1) and exp(a_n - gc_jn) (>= 1): two
  // sets of 16 scaled rows (in the space of T, which is not needed yet) and a 16 x 16 x K fp32 product. A block whose
  // decay spread max_n (a_n - gc_last,n) exceeds 60 keeps one exp per (i, j, n).
  {
    float* s_kq = s_T;             // [16][LD] k exp(gc_i - a)
    float* s_kk = s_T + SUB * LD;  // [16][LD] k exp(a - gc_j)
    __shared__ int s_exact[C / SUB];
    if (tid < C / SUB) s_exact[tid] = 0;
    __syncthreads();
    for (int i = tid; i < (C / SUB) * K; i += 256) {
      const int I = i / K, n = i - I * K;
      if (__fsub_rn(s_gc[(SUB * I) * LD + n], s_gc[(SUB * I + SUB - 1) * LD + n]) > 60.f) s_exact[I] = 1;
    }
    __syncthreads();
    for (int I = 0; I < C / SUB; ++I) {
      if (s_exact[I]) {  // 120 strictly-lower pairs, eight lanes per pair
        for (int pass = 0; pass < 4; ++pass) {
          const int rem_raw = pass * 32 + (tid >> 3);
          const bool valid = rem_raw < 120;  // idle pairs of the last pass compute a clamped pair and store nothing
          const int rem = valid ? rem_raw : 119;
          int i = (int)((sqrtf(8.f * rem + 1.f) + 1.f) * 0.5f);
          while (i * (i + 1) / 2 <= rem) ++i;
          while (i * (i - 1) / 2 > rem) --i;
          const int jj = rem - i * (i - 1) / 2;
          const int ti = SUB * I + i, tj = SUB * I + jj;
          const int l8 = tid & 7;
          float sum = 0.f;
#pragma unroll
          for (int n4 = 0; n4 < K / 32; ++n4) {
            const int n = 4 * l8 + 32 * n4;  // the eight lanes of a pair read 128 consecutive bytes of each row
            const float4 gi = *reinterpret_cast<const float4*>(s_gc + ti * LD + n), gj = *reinterpret_cast<const float4*>(s_gc + tj * LD + n);
            const float4 xi = *reinterpret_cast<const float4*>(s_x + ti * LD + n), xj = *reinterpret_cast<const float4*>(s_x + tj * LD + n);
            sum = fmaf(xi.x * xj.x, __expf(gi.x - gj.x), sum);
            sum = fmaf(xi.y * xj.y, __expf(gi.y - gj.y), sum);
            sum = fmaf(xi.z * xj.z, __expf(gi.z - gj.z), sum);
            sum = fmaf(xi.w * xj.w, __expf(gi.w - gj.w), sum);
          }
          sum += __shfl_xor_sync(0xffffffffu, sum, 1);
          sum += __shfl_xor_sync(0xffffffffu, sum, 2);
          sum += __shfl_xor_sync(0xffffffffu, sum, 4);
          if (l8 == 0 && valid) s_G[ti * 68 + tj] = s_bs[ti] * s_b1[tj] * sum;
        }
        __syncthreads();
        continue;
      }
      for (int i = tid; i < SUB * (K / 4); i += 256) {
        const int rr = i / (K / 4), n = 4 * (i - rr * (K / 4));
        const int t = SUB * I + rr;
        const float4 an = *reinterpret_cast<const float4*>(s_gc + (SUB * I) * LD + n);
        const float4 gt = *reinterpret_cast<const float4*>(s_gc + t * LD + n);
        const float4 xv = *reinterpret_cast<const float4*>(s_x + t * LD + n);
        *reinterpret_cast<float4*>(s_kq + rr * LD + n) = make_float4(__fmul_rn(xv.x, __expf(gt.x - an.x)), __fmul_rn(xv.y, __expf(gt.y - an.y)),
                                                                     __fmul_rn(xv.z, __expf(gt.z - an.z)), __fmul_rn(xv.w, __expf(gt.w - an.w)));
        *reinterpret_cast<float4*>(s_kk + rr * LD + n) = make_float4(__fmul_rn(xv.x, __expf(an.x - gt.x)), __fmul_rn(xv.y, __expf(an.y - gt.y)),
                                                                     __fmul_rn(xv.z, __expf(an.z - gt.z)), __fmul_rn(xv.w, __expf(an.w - gt.w)));
      }
      __syncthreads();
      {  // 16 x 16 x K product on the tensor cores, 3xTF32, as in the A matrix: warp w contracts the channels
         // [K/8 w, K/8 (w + 1)), the eight partial blocks are summed in a fixed order
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int kk = 0; kk < K / 64; ++kk) {
          const int c0 = (K / 8) * warp + 8 * kk + j4, c1 = c0 + 4;
          const float xa[4] = {s_kq[g * LD + c0], s_kq[(g + 8) * LD + c0], s_kq[g * LD + c1], s_kq[(g + 8) * LD + c1]};
          uint32_t ab[4], as_[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ab[e] = tf32_rna(xa[e]);
            as_[e] = tf32_rna(xa[e] - __uint_as_float(ab[e]));
          }
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const float y0 = s_kk[(8 * nt + g) * LD + c0], y1 = s_kk[(8 * nt + g) * LD + c1];
            const uint32_t b0 = tf32_rna(y0), b1 = tf32_rna(y1);
            const uint32_t s0 = tf32_rna(y0 - __uint_as_float(b0)), s1 = tf32_rna(y1 - __uint_as_float(b1));
            mma_tf32(acc[nt], as_[0], as_[1], as_[2], as_[3], b0, b1);
            mma_tf32(acc[nt], ab[0], ab[1], ab[2], ab[3], s0, s1);
            mma_tf32(acc[nt], ab[0], ab[1], ab[2], ab[3], b0, b1);
          }
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          float* pw = s_part + warp * 256;
          pw[g * 16 + 8 * nt + 2 * j4] = acc[nt][0];
          pw[g * 16 + 8 * nt + 2 * j4 + 1] = acc[nt][1];
          pw[(g + 8) * 16 + 8 * nt + 2 * j4] = acc[nt][2];
          pw[(g + 8) * 16 + 8 * nt + 2 * j4 + 1] = acc[nt][3];
        }
        __syncthreads();
        const int i = tid >> 4, jj = tid & 15;
        if (jj < i) {
          float sum = 0.f;
#pragma unroll
          for (int w = 0; w < 8; ++w) sum += s_part[w * 256 + tid];
          const int ti = SUB * I + i;
          s_G[ti * 68 + SUB * I + jj] = s_bs[ti] * s_b1[SUB * I + jj] * sum;
        }
      }
      __syncthreads();
    }
  }

  // ---- off-diagonal blocks: block row I against tokens [0, 16 I), anchored at row 16 I
  for (int I = 1; I < C / SUB; ++I) {
    kda_scaled_rows<T, K>(a, b, c, h, s_gc, s_x, SUB * I, 0, SUB * I, 0, false);        // ke -> rows 0 .. 16I-1
    kda_scaled_rows<T, K>(a, b, c, h, s_gc, s_x, SUB * I, SUB * I, SUB, 48, true);      // kd -> rows 48 .. 63
    __syncthreads();
    // 2 I column tiles of eight tokens x four quarters of the channels = 8 I units of work, dealt to the eight warps
    // (one column tile per warp would leave 8 - 2 I warps idle); the quarter sums are parked in the space of T, which is
    // not needed before the solve, and added in a fixed order.
    for (int u = warp; u < 8 * I; u += 8) {
      const int nt = u >> 2, kq = u & 3;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      const float* ra = s_x + (48 + g) * LD;
      const float* rb = s_x + (56 + g) * LD;
      const float* rn = s_x + (8 * nt + g) * LD;
#pragma unroll
      for (int ks = 0; ks < K / 32; ++ks) {
        const int c0 = 8 * (kq * (K / 32) + ks) + j4, c1 = c0 + 4;
        const float xa[4] = {ra[c0], rb[c0], ra[c1], rb[c1]};
        const float xb[2] = {rn[c0], rn[c1]};
        uint32_t ab[4], as_[4], bb[2], bs_[2];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          ab[e] = tf32_rna(xa[e]);
          as_[e] = tf32_rna(xa[e] - __uint_as_float(ab[e]));
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          bb[e] = tf32_rna(xb[e]);
          bs_[e] = tf32_rna(xb[e] - __uint_as_float(bb[e]));
        }
        mma_tf32(acc, as_[0], as_[1], as_[2], as_[3], bb[0], bb[1]);
        mma_tf32(acc, ab[0], ab[1], ab[2], ab[3], bs_[0], bs_[1]);
        mma_tf32(acc, ab[0], ab[1], ab[2], ab[3], bb[0], bb[1]);
      }
      float* pp = s_T + u * 128;  // [16 rows][8 columns]
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        pp[g * 8 + 2 * j4 + e] = acc[e];
        pp[(g + 8) * 8 + 2 * j4 + e] = acc[2 + e];
      }
    }
    __syncthreads();
    for (int el = tid; el < 256 * I; el += 256) {
      const int i = el / (16 * I), jj = el - i * (16 * I);
      const float* pp = s_T + (4 * (jj >> 3)) * 128 + i * 8 + (jj & 7);
      const float sum = ((pp[0] + pp[128]) + pp[256]) + pp[384];
      const int ia = SUB * I + i;
      s_G[ia * 68 + jj] = s_bs[ia] * s_b1[jj] * sum;
    }
    __syncthreads();
  }
  wy_solve(s_G, s_T);
  // decayed keys k * exp(gc) (the Gram passes are done); then the gc region is free for v
  kda_scaled_rows<T, K>(a, b, c, h, s_gc, s_x, -1, 0, C, 0, false);
  __syncthreads();
  {
    const T* vp = reinterpret_cast<const T*>(a.v);
    constexpr int NIT = C * (V / 8) / 256;
    uint4 raw[NIT];
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int i = tid + 256 * it, t = i / (V / 8), seg = i % (V / 8);
      raw[it] = __ldg(reinterpret_cast<const uint4*>(vp + (((size_t)b * a.T + (size_t)c * C + t) * a.H + h) * V + 8 * seg));
    }
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int i = tid + 256 * it, t = i / (V / 8), seg = i % (V / 8);
      float x[8];
      Act<T>::unpack8(raw[it], x);
      *reinterpret_cast<float4*>(s_vf + t * LDV + 8 * seg) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(s_vf + t * LDV + 8 * seg + 4) = make_float4(x[4], x[5], x[6], x[7]);
    }
  }
  // Row tile mt of W and U contracts over 2 mt + 2 steps of eight tokens: every warp takes the row tiles pr and 3 - pr
  // (five steps on average instead of up to eight) and one quarter of the columns.
  const int pr = warp & 1, qd = warp >> 1;
  const float inv_sw = 1.0f / a.sw[h];
  // ---- W = T diag(beta^sigma) (k exp(gc))  -> w_read codes
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int mt = half == 0 ? pr : 3 - pr;
    constexpr int NTW = K / 32;
    float acc[NTW][4];
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    const int n0 = qd * (K / 4);
    wy_product_split<NTW>(acc, s_T, s_bs, s_x, LD, mt, n0, g, j4);
    const int ia = 16 * mt + g, ib = ia + 8;
#pragma unroll
    for (int nt = 0; nt < NTW; ++nt) {
      const int col = n0 + 8 * nt + 2 * j4;
      const int a0 = q8(Act<T>::round(acc[nt][0]), inv_sw, a.qmax), a1 = q8(Act<T>::round(acc[nt][1]), inv_sw, a.qmax);
      const int b0 = q8(Act<T>::round(acc[nt][2]), inv_sw, a.qmax), b1 = q8(Act<T>::round(acc[nt][3]), inv_sw, a.qmax);
      *reinterpret_cast<uint16_t*>(a.wq + tile * (C * K) + wq_offset(ia, col)) = (uint16_t)((a0 & 0xff) | ((a1 & 0xff) << 8));
      *reinterpret_cast<uint16_t*>(a.wq + tile * (C * K) + wq_offset(ib, col)) = (uint16_t)((b0 & 0xff) | ((b1 & 0xff) << 8));
    }
  }
  __syncthreads();  // v staged by all threads
  // ---- U = T diag(beta^sigma) v (v is exact in TF32)
  T* up = reinterpret_cast<T*>(a.u);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int mt = half == 0 ? pr : 3 - pr;
    constexpr int NTU = V / 32;
    float acc[NTU][4];
#pragma unroll
    for (int nt = 0; nt < NTU; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    const int n0 = qd * (V / 4);
    wy_product<NTU>(acc, s_T, s_bs, s_vf, LDV, mt, n0, g, j4);
    const int ia = 16 * mt + g, ib = ia + 8;
#pragma unroll
    for (int nt = 0; nt < NTU; ++nt) {
      const int col = n0 + 8 * nt + 2 * j4;
      T* uc = up + (tile * V + col) * C;  // [V][C]: the token index contiguous
      uc[ia] = Act<T>::from(acc[nt][0]);
      uc[C + ia] = Act<T>::from(acc[nt][1]);
      uc[ib] = Act<T>::from(acc[nt][2]);
      uc[C + ib] = Act<T>::from(acc[nt][3]);
    }
  }
}

// ------------------------------------------------------------------------------------------------ launchers
int validate_zoo_problem(const lq_zoo_problem* p, bool delta, bool diagonal);

static void fill_diag_args(const lq_zoo_problem* p, const lq_zoo_workspace* ws, DiagArgs& a) {
  a.q = p->q; a.k = p->k; a.v = p->v; a.g = p->g; a.beta = p->beta; a.signs = p->rot_signs;
  a.sq = p->sq; a.sk = p->sk; a.skw = p->skw; a.svl = p->svl; a.svw = p->svw; a.sw = p->sw;
  a.qq = ws->qq; a.kwT = ws->kwT; a.vlT = ws->vlT; a.vwT = ws->vwT; a.wq = ws->wq;
  a.gc = ws->gc; a.genv = ws->genv; a.gcl = ws->gcl; a.fw = ws->fw; a.u = ws->u;
  a.amat = reinterpret_cast<__half*>(ws->amat);
  a.T = p->T; a.H = p->H; a.NT = p->T / p->chunk;
  a.scale = p->scale; a.eta = p->eta; a.sigma = p->sigma; a.tau = p->tau; a.qmax = p->qmax;
}

template <typename KernelT>
static int launch_big_smem(KernelT kern, const char* name, dim3 grid, size_t smem, const DiagArgs& a, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(LQ_ERR_LAUNCH, "%s: cannot opt in to %zu bytes of shared memory: %s", name, smem, cudaGetErrorString(e));
  launch(kern, grid, 256, smem, st, a);
  return check_launch(name);
}

template <typename T, int K, int V>
static int run_diag_T(const lq_zoo_problem* p, const DiagArgs& a, bool delta, int stage, cudaStream_t st) {
  dim3 grid(a.NT, p->B * p->H);
  if (stage == 0) {
    const size_t smem = sizeof(float) * (64 * (K + 4) + 128) + sizeof(uint32_t) * 17 * (K + 2 * V);
    if (delta) return launch_big_smem(zoo_diag_rows_kernel<T, K, V, true>, "zoo_diag_rows_kernel", grid, smem, a, st);
    return launch_big_smem(zoo_diag_rows_kernel<T, K, V, false>, "zoo_diag_rows_kernel", grid, smem, a, st);
  }
  if (stage == 1) {
    const size_t smem = sizeof(float) * (64 * (K + 4) + K + 64) + (size_t)9 * (K / 32) * 512;
    return launch_big_smem(zoo_diag_amat_kernel<T, K>, "zoo_diag_amat_kernel", grid, smem, a, st);
  }
  const size_t smem = sizeof(float) * (64 * ((K + 4) > (V + 8) ? (K + 4) : (V + 8)) + 64 * (K + 4) + 2 * 64 * 68 + 128 + 8 * 256);
  return launch_big_smem(zoo_kda_wy_kernel<T, K, V>, "zoo_kda_wy_kernel", grid, smem, a, st);
}

template <typename T>
static int run_diag_KV(const lq_zoo_problem* p, const DiagArgs& a, bool delta, int stage, cudaStream_t st) {
  if (p->K == 64 && p->V == 64) return run_diag_T<T, 64, 64>(p, a, delta, stage, st);
  if (p->K == 64 && p->V == 128) return run_diag_T<T, 64, 128>(p, a, delta, stage, st);
  if (p->K == 128 && p->V == 64) return run_diag_T<T, 128, 64>(p, a, delta, stage, st);
  if (p->K == 128 && p->V == 128) return run_diag_T<T, 128, 128>(p, a, delta, stage, st);
  return fail(LQ_ERR_UNSUPPORTED, "diagonal decay: K and V must be 64 or 128");
}

// stage 0 = rows, 1 = A matrix, 2 = KDA WY prep
int run_diag_stage(const lq_zoo_problem* p, const lq_zoo_workspace* ws, bool delta, int stage, cudaStream_t st) {
  DiagArgs a;
  fill_diag_args(p, ws, a);
  if (p->act_dtype == LQ_F16) return run_diag_KV<__half>(p, a, delta, stage, st);
  if (p->act_dtype == LQ_BF16) return run_diag_KV<__nv_bfloat16>(p, a, delta, stage, st);
  return fail(LQ_ERR_UNSUPPORTED, "diagonal decay: activation dtype must be f16 or bf16");
}

}  // namespace lq

extern "C" int lq_zoo_diag_rows(const lq_zoo_problem* p, const lq_zoo_workspace* ws, lq_stream stream) {
  const bool delta = p && p->beta != nullptr;
  if (int e = lq::validate_zoo_problem(p, delta, true)) return e;
  if (!ws) return lq::fail(LQ_ERR_NULL, "diag rows: workspace descriptor is null");
  return lq::run_diag_stage(p, ws, delta, 0, (cudaStream_t)stream);
}
extern "C" int lq_zoo_diag_amat(const lq_zoo_problem* p, const lq_zoo_workspace* ws, lq_stream stream) {
  const bool delta = p && p->beta != nullptr;
  if (int e = lq::validate_zoo_problem(p, delta, true)) return e;
  if (!ws) return lq::fail(LQ_ERR_NULL, "diag amat: workspace descriptor is null");
  return lq::run_diag_stage(p, ws, delta, 1, (cudaStream_t)stream);
}
extern "C" int lq_zoo_kda_wy(const lq_zoo_problem* p, const lq_zoo_workspace* ws, lq_stream stream) {
  if (int e = lq::validate_zoo_problem(p, true, true)) return e;
  if (!ws) return lq::fail(LQ_ERR_NULL, "kda wy: workspace descriptor is null");
  return lq::run_diag_stage(p, ws, true, 2, (cudaStream_t)stream);
}
