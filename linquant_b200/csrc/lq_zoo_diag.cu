// Diagonal (per-channel) decay cells: GLA (linear family) and KDA (delta family).
//
// Three chunk-parallel kernels, one CTA per (batch*head, chunk):
//   rows   chunk-local cumulative log-decay per channel (double accumulate), log envelope, pre-decayed q_read codes,
//          gated k_write codes (Omega * s^-eta), and for the linear family the v_local / v_write codes
//   amat   the intra-chunk matrix A in 16-token secondary chunks: off-diagonal blocks as INT8 MMAs on operands
//          re-scaled around the block's anchor row (optionally rotated by a signed Hadamard on fp16-rounded values),
//          diagonal blocks as tensor-core products of the dequantised codes times their weights around the block's first
//          row, three bf16 pieces each (an fp32 reduction with one exp per (i, j, channel) where the decay is too strong)
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

template <int K, int BATCH>
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
// Work items of a warp: 32 tokens x 32 channels of q and k, or of v; a thread takes four tokens x eight channels, so that the
// transposed codes are whole words and go straight to global memory (32 contiguous bytes per channel). The q / k rows travel
// during the decay scan. Bound by HBM at the KDA configuration, by the scan's latency where few CTAs run. The kernel before it (codes one at a time,
// transposed through shared memory, rows requested after the scan) took 892 us for 256 (b, h) x 128 chunks at K = 128 (KDA)
// and 88 us for 32 x 64 with K = V = 128 (GLA); this one 584
// (0.98 of the time its 3.8 GB take at 6.55 TB/s) and 56.
template <int K, int V>
constexpr size_t diag_rows_smem() { return sizeof(float) * (64 * (K + 4) + 128 + K + 2 * V); }

template <typename T, int K, int V, bool DELTA>
__global__ void __launch_bounds__(256, 3) zoo_diag_rows_kernel(DiagArgs a) {
  pdl_enter();
  constexpr int C = 64, LD = K + 4, NQK = K / 16;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* s_gc = reinterpret_cast<float*>(smem_raw);
  float* s_le = s_gc + C * LD;
  float* s_hw = s_le + C;
  float* s_ikw = s_hw + C;  // [K] 1 / scale
  float* s_ivl = s_ikw + K;  // [V]
  float* s_ivw = s_ivl + V;  // [V]

  const int c = blockIdx.x, bh = blockIdx.y;
  const int b = bh / a.H, h = bh % a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t tile = (size_t)bh * a.NT + c;
  const size_t tok0 = ((size_t)b * a.T + (size_t)c * C) * a.H + h;
  const float e_hw = (1.f - a.sigma) * a.tau;
  const int lt = 4 * (lane >> 2), ln = 8 * (lane & 3);  // the thread's first token and channel in an item

  // the raw log-decays of the chunk, and the rows of the warp's q / k item
  for (int i = tid; i < C * (K / 4); i += 256) {
    const int t = i / (K / 4), n = 4 * (i % (K / 4));
    cp_async16(s_gc + t * LD + n, a.g + (tok0 + (size_t)t * a.H) * K + n);
  }
  cp_async_commit();
  uint4 rq[4], rk[4];
  if (warp < NQK) {
    const int t0 = 32 * (warp & 1) + lt, n0 = 32 * (warp >> 1) + ln;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t row = (tok0 + (size_t)(t0 + i) * a.H) * K + n0;
      rq[i] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.q) + row));
      rk[i] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.k) + row));
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // one thread per channel scans in double; the others form the reciprocal scales
  if (tid < K) {
    double acc = 0.0;
    float f = 0.f;
#pragma unroll 1
    for (int t0 = 0; t0 < C; t0 += 16) {
      float x[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) x[t] = s_gc[(t0 + t) * LD + tid];
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        acc += (double)x[t];
        f = (float)acc;
        s_gc[(t0 + t) * LD + tid] = f;
      }
    }
    a.gcl[tile * K + tid] = expf(f);
  } else {
    for (int i = tid - K; i < K; i += 256 - K) s_ikw[i] = 1.0f / a.skw[h * K + i];
    if (!DELTA) {
      for (int i = tid - K; i < V; i += 256 - K) {
        s_ivl[i] = 1.0f / a.svl[h * V + i];
        s_ivw[i] = 1.0f / a.svw[h * V + i];
      }
    } else if (tid >= 256 - C) {
      const int t = tid - (256 - C);
      s_hw[t] = pow_exact01(a.beta[tok0 + (size_t)t * a.H], e_hw);
    }
  }
  __syncthreads();
  for (int i = tid; i < C * (K / 4); i += 256) {
    const int t = i / (K / 4), c4 = i % (K / 4);
    reinterpret_cast<float4*>(a.gc + (tile * C + t) * K)[c4] = *reinterpret_cast<const float4*>(s_gc + t * LD + 4 * c4);
  }
  if (a.eta != 0.f) {  // log envelope: with eta = 0 every gate is 1
    for (int tt = 0; tt < 8; ++tt) {
      const int t = 8 * warp + tt;
      float m = -INFINITY;
      for (int n = lane; n < K; n += 32) m = fmaxf(m, s_gc[(C - 1) * LD + n] - s_gc[t * LD + n]);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
      if (lane == 0) {
        s_le[t] = a.eta * m;
        a.genv[tile * C + t] = expf(a.eta * m);
      }
    }
    __syncthreads();
  } else if (tid < C) {
    a.genv[tile * C + tid] = 1.f;
  }

  // words of four tokens from codes of channel pairs: channels n, n + 1 of tokens 0, 1 and of tokens 2, 3
  auto put = [&](int8_t* dst, const F2 (&x)[4], F2 inv) {
    const uint32_t lo = codes4<false>(x[0], x[1], inv, a.qmax), hi = codes4<false>(x[2], x[3], inv, a.qmax);
    *reinterpret_cast<uint32_t*>(dst) = __byte_perm(lo, hi, 0x6420);
    *reinterpret_cast<uint32_t*>(dst + C) = __byte_perm(lo, hi, 0x7531);
  };
  if (warp < NQK) {
    const int t0 = 32 * (warp & 1) + lt, n0 = 32 * (warp >> 1) + ln;
    const float inv_sq = 1.0f / a.sq[h];
    const F2 inv(inv_sq, inv_sq), scale(a.scale, a.scale);
    F2 gl[4], y[4][4];  // [token][channel pair]
#pragma unroll
    for (int p = 0; p < 4; ++p) gl[p] = F2(s_gc[(C - 1) * LD + n0 + 2 * p], s_gc[(C - 1) * LD + n0 + 2 * p + 1]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = t0 + i;
      float x[8], gv[8];
      *reinterpret_cast<float4*>(gv) = *reinterpret_cast<const float4*>(s_gc + t * LD + n0);
      *reinterpret_cast<float4*>(gv + 4) = *reinterpret_cast<const float4*>(s_gc + t * LD + n0 + 4);
      Act<T>::unpack8(rq[i], x);
      uint32_t cd[2];
#pragma unroll
      for (int eh = 0; eh < 2; ++eh) {
        const int e = 4 * eh;
        cd[eh] = codes4<false>(mul2(mul2(F2(x[e], x[e + 1]), exp_pair(F2(gv[e], gv[e + 1]))), scale),
                               mul2(mul2(F2(x[e + 2], x[e + 3]), exp_pair(F2(gv[e + 2], gv[e + 3]))), scale), inv, a.qmax);
      }
      *reinterpret_cast<uint2*>(a.qq + (tile * C + t) * K + n0) = make_uint2(cd[0], cd[1]);
      Act<T>::unpack8(rk[i], x);
      if (DELTA && e_hw != 0.f) {
        const float hw = s_hw[t];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = Act<T>::round(__fmul_rn(x[e], hw));
      }
      const float ele = a.eta != 0.f ? s_le[t] : 0.f;
#pragma unroll
      for (int p = 0; p < 4; ++p)
        y[i][p] = mul2(F2(x[2 * p], x[2 * p + 1]), exp_pair(sub2(sub2(gl[p], F2(gv[2 * p], gv[2 * p + 1])), F2(ele, ele))));
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const F2 w[4] = {y[0][p], y[1][p], y[2][p], y[3][p]};
      put(a.kwT + (tile * K + n0 + 2 * p) * C + t0, w, F2(s_ikw[n0 + 2 * p], s_ikw[n0 + 2 * p + 1]));
    }
  }
  if (const int u = (warp + NQK) & 7; !DELTA && u < V / 16) {  // K = 64: the warps without a q / k item first
    const int t0 = 32 * (u & 1) + lt, n0 = 32 * (u >> 1) + ln;
    uint4 rv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) rv[i] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.v) + (tok0 + (size_t)(t0 + i) * a.H) * V + n0));
    float x[4][8], fv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      Act<T>::unpack8(rv[i], x[i]);
      fv[i] = a.eta != 0.f ? expf(s_le[t0 + i]) : 1.f;
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      F2 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = F2(x[i][2 * p], x[i][2 * p + 1]);
      put(a.vlT + (tile * V + n0 + 2 * p) * C + t0, w, F2(s_ivl[n0 + 2 * p], s_ivl[n0 + 2 * p + 1]));
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = mul2(w[i], F2(fv[i], fv[i]));
      put(a.vwT + (tile * V + n0 + 2 * p) * C + t0, w, F2(s_ivw[n0 + 2 * p], s_ivw[n0 + 2 * p + 1]));
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
// split in the product loop: 42 k warp instructions and 27 block barriers per chunk) took 2070 us for 256 (b, h) x 128 chunks at
// K = 128, this one 1637; with pairwise exponentials, the channel loop of the diagonal blocks rolled (unrolled, waiting for instructions
// was the first stall) and one form of the code rule 1228; 1233 since a diagonal block is summed from one fresh accumulator per 32
// channels (sums in one accumulator throughout cut off bits: up to 1.5 times as many fp16 results beside the right one).
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
    uint4 nq[2], nk[2];  // the rows of the next 32 channels
    const T* rowp[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      rowp[r][0] = qp + grow(t0 + g + 8 * r);
      rowp[r][1] = kp + grow(t0 + g + 8 * r);
      nq[r] = __ldg(reinterpret_cast<const uint4*>(rowp[r][0]));
      nk[r] = __ldg(reinterpret_cast<const uint4*>(rowp[r][1]));
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
#pragma unroll 1  // 600 instructions a pass: unrolled, the kernel waits for its instructions
      for (int m = 0; m < M; ++m) {
        float an[8];
        lds8(s_gc + t0 * LD + 32 * m + 8 * j, an);
        uint32_t qh[2][4], qm[2][4], ql[2][4], kh[2][4], km[2][4], kl[2][4];  // [row half][pair of channels]
        const uint4 rq[2] = {nq[0], nq[1]}, rk[2] = {nk[0], nk[1]};
        if (m + 1 < M) {
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            nq[r] = __ldg(reinterpret_cast<const uint4*>(rowp[r][0] + 32 * (m + 1)));
            nk[r] = __ldg(reinterpret_cast<const uint4*>(rowp[r][1] + 32 * (m + 1)));
          }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int t = t0 + g + 8 * r;
          float x[8], gv[8];
          F2 e1[4];
          lds8(s_gc + t * LD + 32 * m + 8 * j, gv);
          Act<T>::unpack8(rq[r], x);
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            e1[p] = sub2(F2(gv[2 * p], gv[2 * p + 1]), F2(an[2 * p], an[2 * p + 1]));
            split3_pair(mul2(code_pair(mul2(F2(x[2 * p], x[2 * p + 1]), F2(a.scale, a.scale)), fq, a.qmax), exp_pair(e1[p])), qh[r][p], qm[r][p], ql[r][p]);
          }
          key(rk[r], t, x);
#pragma unroll
          for (int p = 0; p < 4; ++p)
            split3_pair(mul2(code_pair(F2(x[2 * p], x[2 * p + 1]), fk, a.qmax), exp_pair(mul2(e1[p], F2(-1.f, -1.f)))), kh[r][p], km[r][p], kl[r][p]);
        }
        // The tensor core cuts off what falls below the last bit of its accumulator: the products go small to big into a fresh
        // one per 32 channels (only the two biggest meet a full sum), and the passes are added in fp32.
        float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        auto mma = [&](const uint32_t (&qa)[2][4], const uint32_t (&kb)[2][4]) {
#pragma unroll
          for (int p = 0; p < 4; p += 2)
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) mma_bf16(d[nt], qa[0][p], qa[1][p], qa[0][p + 1], qa[1][p + 1], kb[nt][p], kb[nt][p + 1]);
        };
        mma(ql, kh);
        mma(qh, kl);
        mma(qm, km);
        mma(qm, kh);
        mma(qh, km);
        mma(qh, kh);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[nt][i] += d[nt][i];
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
          for (int e = 0; e < 8; e += 2)
            mul2(mul2(F2(x[r][e], x[r][e + 1]), exp_pair(sub2(F2(gv[e], gv[e + 1]), F2(an[e], an[e + 1])))), F2(a.scale, a.scale)).get(x[r][e], x[r][e + 1]);
        } else {
          if (use_hw) {
            const float hw = s_hw[t];
#pragma unroll
            for (int e = 0; e < 8; ++e) x[r][e] = Act<T>::round(__fmul_rn(x[r][e], hw));
          }
#pragma unroll
          for (int e = 0; e < 8; e += 2)
            mul2(F2(x[r][e], x[r][e + 1]), exp_pair(sub2(F2(an[e], an[e + 1]), F2(gv[e], gv[e + 1])))).get(x[r][e], x[r][e + 1]);
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
          w[r][eh] = codes4<false>(y0, y1, inv, a.qmax);
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
// secondary chunks like the A matrix: for block row I the weight factors around its first row a = 16 I,
//   kd[i,n] = k[i,n] exp(gc[i,n] - gc[a,n])  (<= 1),   ke[j,n] = k[j,n] exp(gc[a,n] - gc[j,n])  (<= 1 for the earlier blocks),
// each split into three bf16 pieces (exact) and contracted in six products on the tensor cores. A warp takes a quarter of the
// channels and block rows 0 and 3, or 1 and 2: seven operand tiles each, made in the registers of the fragments that
// contract them (a lane holds K/16 consecutive channels of its two rows), and the four quarters are added in a fixed order.
// W = T diag(beta^sigma) (k exp(gc)) and U = T diag(beta^sigma) v follow on the same three-piece products (lq_wy.cuh).
// Bound by instruction issue. The kernel before it (operands through shared memory once per block row, 3xTF32 with the split
// in the product loop, 30 block barriers: 58 k warp instructions a chunk) took 3480 us for 256 (b, h) x 128 chunks at
// K = V = 128; this one 1692 (1826 before its exponentials and the codes of W were taken in pairs).
template <int K, int V>
struct KdaWySmem {
  static constexpr int LD = K + 4, LDR = K + 8, LDV = V + 8;  // fp32 log-decays, raw k rows, raw v rows
  static constexpr int kGc = 0, kK = kGc + 4 * 64 * LD, kV = kK + 2 * 64 * LDR;
  static constexpr int kWork = kV + 2 * 64 * LDV;  // quarter sums of the Gram blocks; then G | T; then the fragments of T in G's place
  static constexpr int kBeta = kWork + 4 * 10 * 1024, kBytes = kBeta + 4 * 128;
};
template <int K, int V>
constexpr size_t kda_wy_smem() { return KdaWySmem<K, V>::kBytes; }

template <typename T, int K, int V>
__global__ void __launch_bounds__(256, 2) zoo_kda_wy_kernel(DiagArgs a) {
  pdl_enter();
  typedef KdaWySmem<K, V> S;
  constexpr int C = 64, LD = S::LD, LDR = S::LDR, LDV = S::LDV, SUB = 16, CH = K / 16, KS = K / 64;
  static_assert(2 * C * 68 * 4 <= 4 * 10 * 1024 && 30 * 512 <= C * 68 * 4, "aliases of the work area");
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* s_gc = reinterpret_cast<float*>(smem_raw + S::kGc);
  T* s_k = reinterpret_cast<T*>(smem_raw + S::kK);
  T* s_v = reinterpret_cast<T*>(smem_raw + S::kV);
  float4* s_part = reinterpret_cast<float4*>(smem_raw + S::kWork);  // [quarter][block][n-tile][lane]
  float* s_G = reinterpret_cast<float*>(smem_raw + S::kWork);
  float* s_T = s_G + C * 68;
  uint4* s_frag = reinterpret_cast<uint4*>(smem_raw + S::kWork);
  float* s_bs = reinterpret_cast<float*>(smem_raw + S::kBeta);
  float* s_b1 = s_bs + C;

  const int c = blockIdx.x, bh = blockIdx.y;
  const int b = bh / a.H, h = bh % a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, j = lane & 3;
  const size_t tile = (size_t)bh * a.NT + c;
  const size_t tok0 = ((size_t)b * a.T + (size_t)c * C) * a.H + h;

  for (int i = tid; i < C * K / 4; i += 256) {
    const int t = i / (K / 4), n = 4 * (i % (K / 4));
    cp_async16(s_gc + t * LD + n, a.gc + (tile * C + t) * K + n);
  }
  for (int i = tid; i < C * K / 8; i += 256) {
    const int t = i / (K / 8), n = 8 * (i % (K / 8));
    cp_async16(s_k + t * LDR + n, reinterpret_cast<const T*>(a.k) + (tok0 + (size_t)t * a.H) * K + n);
  }
  cp_async_commit();
  for (int i = tid; i < C * V / 8; i += 256) {
    const int t = i / (V / 8), n = 8 * (i % (V / 8));
    cp_async16(s_v + t * LDV + n, reinterpret_cast<const T*>(a.v) + (tok0 + (size_t)t * a.H) * V + n);
  }
  cp_async_commit();
  if (tid < C) {
    const float bt = a.beta[tok0 + (size_t)tid * a.H];
    s_bs[tid] = pow_exact01(bt, a.sigma);
    s_b1[tid] = pow_exact01(bt, 1.f - a.sigma);
    a.fw[tile * C + tid] = pow_exact01(bt, (1.f - a.sigma) * (1.f - a.tau));
  }
  cp_async_wait<1>();
  __syncthreads();

  // ---- Gram blocks, one quarter of the channels
  {
    const int n0 = (K / 4) * (warp & 3) + CH * j;
    auto ldg = [&](int t, float (&x)[CH]) {
#pragma unroll
      for (int e = 0; e < CH; e += 4) *reinterpret_cast<float4*>(x + e) = *reinterpret_cast<const float4*>(s_gc + t * LD + n0 + e);
    };
    auto ldk = [&](int t, float (&x)[CH]) {
      if constexpr (CH == 8) {
        Act<T>::unpack8(*reinterpret_cast<const uint4*>(s_k + t * LDR + n0), x);
      } else {
        const uint2 w = *reinterpret_cast<const uint2*>(s_k + t * LDR + n0);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = Act<T>::get(e < 2 ? w.x : w.y, e & 1);
      }
    };
    for (int half = 0; half < 2; ++half) {
      const int I = warp < 4 ? 3 * half : 1 + half;
      float an[CH];
      ldg(SUB * I, an);
      uint32_t ah[2][CH / 2], am[2][CH / 2], al[2][CH / 2];  // [row half][pair of channels]
      float lowest = 0.f;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float x[CH], gv[CH];
        ldg(SUB * I + g + 8 * r, gv);
        ldk(SUB * I + g + 8 * r, x);
#pragma unroll
        for (int p = 0; p < CH / 2; ++p) {
          const F2 d = sub2(F2(gv[2 * p], gv[2 * p + 1]), F2(an[2 * p], an[2 * p + 1]));
          float d0, d1;
          d.get(d0, d1);
          lowest = fminf(lowest, fminf(d0, d1));
          split3_pair(mul2(F2(x[2 * p], x[2 * p + 1]), exp_pair(d)), ah[r][p], am[r][p], al[r][p]);
        }
      }
      // the factors of the diagonal block stay in fp32's range unless the decay across it is beyond e^60
      const bool exact = __any_sync(0xffffffffu, lowest < -60.f);
      for (int J = 0; J <= I; ++J) {
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        if (J < I || !exact) {
          uint32_t bh_[2][CH / 2], bm[2][CH / 2], bl[2][CH / 2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            float x[CH], gv[CH];
            ldg(SUB * J + g + 8 * r, gv);
            ldk(SUB * J + g + 8 * r, x);
#pragma unroll
            for (int p = 0; p < CH / 2; ++p) {
              const F2 w = exp_pair(sub2(F2(an[2 * p], an[2 * p + 1]), F2(gv[2 * p], gv[2 * p + 1])));
              split3_pair(mul2(F2(x[2 * p], x[2 * p + 1]), w), bh_[r][p], bm[r][p], bl[r][p]);
            }
          }
          auto mma = [&](const uint32_t (&qa)[2][CH / 2], const uint32_t (&kb)[2][CH / 2], int p) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) mma_bf16(acc[nt], qa[0][p], qa[1][p], qa[0][p + 1], qa[1][p + 1], kb[nt][p], kb[nt][p + 1]);
          };
#pragma unroll
          for (int p = 0; p < CH / 2; p += 2) {
            mma(al, bh_, p);
            mma(ah, bl, p);
            mma(am, bm, p);
            mma(am, bh_, p);
            mma(ah, bm, p);
            mma(ah, bh_, p);
          }
        } else {
          // one exp per (i, j, channel), a lane for each of its eight (i, j) of the accumulator layout
          for (int n = (K / 4) * (warp & 3); n < (K / 4) * (warp & 3) + K / 4; ++n) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int ti = SUB * I + g + 8 * (e >> 1), tj = SUB * I + 8 * nt + 2 * j + (e & 1);
                const float w = tj < ti ? __expf(s_gc[ti * LD + n] - s_gc[tj * LD + n]) : 0.f;
                acc[nt][e] = fmaf(Act<T>::to(s_k[ti * LDR + n]) * Act<T>::to(s_k[tj * LDR + n]), w, acc[nt][e]);
              }
          }
        }
        const int blk = I * (I + 1) / 2 + J;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
          s_part[(((warp & 3) * 10 + blk) * 2 + nt) * 32 + lane] = make_float4(acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3]);
      }
    }
  }
  __syncthreads();
  {  // 10 blocks x 2 n-tiles x 32 lanes, summed in registers: G takes the place of the quarter sums
    float4 sum[3];
#pragma unroll
    for (int it = 0; it < 3; ++it) {
      const int f = tid + 256 * it;
      if (f < 640) {
        const float4 p0 = s_part[f], p1 = s_part[640 + f], p2 = s_part[1280 + f], p3 = s_part[1920 + f];
        sum[it] = make_float4(((p0.x + p1.x) + p2.x) + p3.x, ((p0.y + p1.y) + p2.y) + p3.y, ((p0.z + p1.z) + p2.z) + p3.z,
                              ((p0.w + p1.w) + p2.w) + p3.w);
      }
    }
    cp_async_wait<0>();  // v: seen by all after the barriers of the solve
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 3; ++it) {
      const int f = tid + 256 * it;
      if (f < 640) {
        const int blk = f >> 6, I = blk < 1 ? 0 : blk < 3 ? 1 : blk < 6 ? 2 : 3, J = blk - I * (I + 1) / 2;
        const int i = SUB * I + g, jj = SUB * J + 8 * ((f >> 5) & 1) + 2 * j;
        const float c0 = s_b1[jj], c1 = s_b1[jj + 1];
        *reinterpret_cast<float2*>(s_G + i * 68 + jj) = make_float2(jj < i ? s_bs[i] * c0 * sum[it].x : 0.f, jj + 1 < i ? s_bs[i] * c1 * sum[it].y : 0.f);
        *reinterpret_cast<float2*>(s_G + (i + 8) * 68 + jj) =
            make_float2(jj < i + 8 ? s_bs[i + 8] * c0 * sum[it].z : 0.f, jj + 1 < i + 8 ? s_bs[i + 8] * c1 * sum[it].w : 0.f);
      }
    }
  }
  __syncthreads();
  wy_solve(s_G, s_T);
  wy_fragments(s_T, s_bs, s_frag, warp, lane);  // in the place of G
  __syncthreads();
  // ---- W = T diag(beta^sigma) (k exp(gc))  -> w_read codes
  {
    const int n0 = (K / 8) * warp;
    float acc[4][KS][4];
    wy_product3<KS, 3>(acc, s_frag, lane, [&](int ks, uint32_t (&bp)[3][KS][2]) {
      uint32_t raw[KS][2];
      wy_ldmatrix<KS>(raw, s_k + 16 * ks * LDR + n0, LDR, lane);
#pragma unroll
      for (int nt = 0; nt < KS; ++nt)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const float* gp = s_gc + (16 * ks + 8 * s + 2 * j) * LD + n0 + 8 * nt + g;
          split3_pair(mul2(F2(Act<T>::get(raw[nt][s], 0), Act<T>::get(raw[nt][s], 1)), exp_pair(F2(gp[0], gp[LD]))), bp[0][nt][s], bp[1][nt][s],
                      bp[2][nt][s]);
        }
    });
    wy_store_w<T, KS>(acc, a.wq + tile * (C * K), n0, 1.0f / a.sw[h], a.qmax, lane);
  }
  // ---- U = T diag(beta^sigma) v
  wy_u<T, V>(s_frag, s_v, LDV, reinterpret_cast<T*>(a.u) + tile * (size_t)(V * C), warp, lane);
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
static int launch_diag(KernelT kern, const char* name, dim3 grid, size_t smem, const DiagArgs& a, cudaStream_t st) {
  const cudaError_t e = launch_opt_in(kern, grid, 256, smem, st, a);
  if (e != cudaSuccess) return fail(LQ_ERR_LAUNCH, "%s (%zu bytes of shared memory): %s", name, smem, cudaGetErrorString(e));
  return check_launch(name);
}

template <typename T, int K, int V>
static int run_diag_T(const lq_zoo_problem* p, const DiagArgs& a, bool delta, int stage, cudaStream_t st) {
  dim3 grid(a.NT, p->B * p->H);
  if (stage == 0) {
    constexpr size_t smem = diag_rows_smem<K, V>();
    if (delta) return launch_diag(zoo_diag_rows_kernel<T, K, V, true>, "zoo_diag_rows_kernel", grid, smem, a, st);
    return launch_diag(zoo_diag_rows_kernel<T, K, V, false>, "zoo_diag_rows_kernel", grid, smem, a, st);
  }
  if (stage == 1) {
    const size_t smem = sizeof(float) * (64 * (K + 4) + K + 64) + (size_t)9 * (K / 32) * 512;
    return launch_diag(zoo_diag_amat_kernel<T, K>, "zoo_diag_amat_kernel", grid, smem, a, st);
  }
  return launch_diag(zoo_kda_wy_kernel<T, K, V>, "zoo_kda_wy_kernel", grid, kda_wy_smem<K, V>(), a, st);
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
