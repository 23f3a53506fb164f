// Delta-rule family (DeltaNet / Gated DeltaNet, none or scalar decay): WY prologue and the chunk-serial state pass.
//
// Prologue (one CTA per (batch*head, chunk), parallel over chunks):
//   q, k rows as in the linear prologue (rescale, Walsh-Hadamard rotation, rounding, codes); the readout/write
//   key is Hw = round(beta^((1-sigma)tau) * k). Then the WY representation of the chunk in fp32-grade arithmetic:
//     G = tril( (beta^sigma k)(beta^(1-sigma) k)^T * exp(gc_i - gc_j), -1 )      fp16 / bf16 MMA on the keys as they are
//     T = (I + G)^-1                                                             blocked inverse (lq_wy.cuh)
//     W = T diag(beta^sigma exp(gc)) k ,  U = T diag(beta^sigma) v              bf16 MMA, the left factor in three pieces
//   W is rounded to the activation dtype and quantised per head (w_read codes); U is stored in the activation dtype.
//   k and v are one bf16 piece (bf16) or two (fp16), the fp32 left factor T diag(.) three (8 + 8 + 8 bits): every product is
//   exact and only the fp32 accumulation rounds.
//
// State pass (groups of warps own 16 value channels of a (batch, head), serial over chunks, fp32 carry [v,k] in registers):
//   hq = q8(carry)  -> stored state and MMA operand;  ws = wq . hq (INT8 MMA);  E = (U - deq(ws)) * fw
//   e_local codes from the activation-rounded E, e_write codes from E * Omega^eta;  carry <- gamma carry + deq(ew^T kw)
//
// Reference arithmetic: zoo/gated_delta_rule.py:20-47 (_prep), :51-115 (_delta_state_body);
// reference.py:202-229 (_chunk_delta).
#include <type_traits>

#include "lq_tc.cuh"
#include "lq_wy.cuh"
#include "lq_zoo_rows.cuh"

namespace lq {

struct DeltaPrepArgs {
  PrologueArgs pro;
  const float *beta, *sw;
  int8_t* wq;
  void* u;
  float *fw, *genv;
  float sigma, tau;
};

// Shared memory: the rotated keys (activation dtype, or fp32 where D_QK is given without a rotation and they are not rounded),
// the raw values, and a work area that holds G and T = (I + G)^-1, then the fragments of T diag(cw) for W and U.
template <typename T, int K, int V, bool KF32>
struct DeltaPrepSmem {
  typedef typename std::conditional<KF32, float, T>::type KT;
  static constexpr int LDK = K + (KF32 ? 4 : 8), LDV = V + 8;
  static constexpr int kK = 4 * (6 * 64 + 4 * K), kV = kK + (int)sizeof(KT) * 64 * LDK, kWork = kV + 2 * 64 * LDV;
  static constexpr int kBytes = kWork + 4 * 2 * 64 * 68;
};

// One CTA per chunk, four steps between block barriers:
//   1  four warps a 16-token tile of k each, four of q: D_QK, Hadamard rotation (sixteen slots of an m16n8k16 product with
//      the +-1 matrix, the rest a butterfly between the lane's own registers; fp32 operands as three bf16 pieces, exact),
//      rounding; q codes out, k to shared memory
//   2  k codes from shared memory (a thread holds four tokens x eight channels, so that the transposed codes are whole words)
//      and the Gram blocks (exact products of 16-bit keys, fp32 accumulation)
//   3  the blocked inverse
//   4  W and U on three-piece products (lq_wy.cuh)
// Bound by instruction issue and the latency of the inverse. The kernel before it (shuffle Hadamard, fp32 staging, TF32
// operands split in the product loop; 112 KB of shared memory) took 774 us for 64 (b, h) x 128 chunks at K = V = 128
// with D_QK; this one 490. Three CTAs per SM at 80 registers spill and gave 867 against 851 us for the whole call.
template <typename T, int K, int V, bool KF32>
__global__ void __launch_bounds__(256, 2) zoo_prologue_delta_kernel(DeltaPrepArgs d) {
  pdl_enter();
  typedef DeltaPrepSmem<T, K, V, KF32> S;
  typedef typename S::KT KT;
  constexpr int C = kChunk, LDK = S::LDK, LDV = S::LDV, M = K / 32, KS = K / 64;
  constexpr bool F16 = std::is_same<T, __half>::value;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* s_gc = reinterpret_cast<float*>(smem_raw);
  float* s_fk = s_gc + C;
  float* s_bs = s_fk + C;
  float* s_b1 = s_bs + C;
  float* s_hw = s_b1 + C;
  float* s_cwW = s_hw + C;   // beta^sigma * exp(gc)
  float* s_ikw = s_cwW + C;  // [K] 1 / k_write scale
  float* s_sgn = s_ikw + K;  // [K] rotation signs / sqrt(K)
  float* s_dq = s_sgn + K;   // [2][K] D_QK of q, of k
  KT* s_k = reinterpret_cast<KT*>(smem_raw + S::kK);
  T* s_v = reinterpret_cast<T*>(smem_raw + S::kV);
  float* s_G = reinterpret_cast<float*>(smem_raw + S::kWork);
  float* s_T = s_G + C * 68;
  uint4* s_frag = reinterpret_cast<uint4*>(smem_raw + S::kWork);  // W's fragments, then U's

  const PrologueArgs& a = d.pro;
  const int c = blockIdx.x, bh = blockIdx.y;
  const int b = bh / a.H, h = bh % a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, j = lane & 3;
  const size_t tile = (size_t)bh * a.NT + c;
  const size_t tok0 = ((size_t)b * a.T + (size_t)c * C) * a.H + h;
  const float e_hw = (1.f - d.sigma) * d.tau;
  const bool rot = !KF32 && a.signs != nullptr, dqk = KF32 || a.dqk != nullptr;

  // every global row of the CTA is requested before the first is used
  const bool isq = warp >= 4;
  const int t0 = 16 * (warp & 3);
  const T* src = reinterpret_cast<const T*>(isq ? a.q : a.k);
  uint4 raw[2][M];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m)
      raw[r][m] = __ldg(reinterpret_cast<const uint4*>(src + (tok0 + (size_t)(t0 + g + 8 * r) * a.H) * K + 32 * m + 8 * j));
  for (int i = tid; i < C * V / 8; i += 256) {
    const int t = i / (V / 8), n = 8 * (i % (V / 8));
    cp_async16(s_v + t * LDV + n, reinterpret_cast<const T*>(a.v) + (tok0 + (size_t)t * a.H) * V + n);
  }
  cp_async_commit();
  if (warp == 0) {
    if (a.g != nullptr) {
      chunk_decay_scan(a.g, b, c, h, a.T, a.H, s_gc);
    } else {
      s_gc[lane] = 0.f;
      s_gc[lane + 32] = 0.f;
    }
  }
  if (tid >= 256 - K) {
    const int n = tid - (256 - K);
    s_ikw[n] = 1.0f / a.skw[h * K + n];
    s_sgn[n] = rot ? a.signs[n] * (K == 64 ? 0.125f : 0.08838834764831845f) : 1.f;
    const float dm = dqk ? a.dqk[h * K + n] : 1.f;
    s_dq[n] = dm;
    s_dq[K + n] = 1.0f / dm;
  }
  __syncthreads();
  if (tid < C) {
    const float dd = s_gc[C - 1] - s_gc[tid];
    s_fk[tid] = a.g ? expf((1.0f - a.eta) * dd) : 1.0f;
    a.gc[tile * C + tid] = s_gc[tid];
    d.genv[tile * C + tid] = a.g ? expf(a.eta * dd) : 1.0f;
    const float bt = d.beta[tok0 + (size_t)tid * a.H];
    const float bs = pow_exact01(bt, d.sigma);
    s_bs[tid] = bs;
    s_b1[tid] = pow_exact01(bt, 1.f - d.sigma);
    s_hw[tid] = pow_exact01(bt, e_hw);
    s_cwW[tid] = a.g ? bs * expf(s_gc[tid]) : bs;
    d.fw[tile * C + tid] = pow_exact01(bt, (1.f - d.sigma) * (1.f - d.tau));
  }

  // ---- 1. rows of q (codes) or k (to shared memory)
  {
    const uint32_t one = F16 && !dqk ? 0x3C00u : 0x3F80u;
    const uint32_t had = [&]() {  // (-1)^popc(s & n) for slots s = 2j, 2j + 1 and column n = g
      const uint32_t s0 = one | ((__popc((2 * j) & g) & 1) << 15), s1 = one | ((__popc((2 * j + 1) & g) & 1) << 15);
      return s0 | (s1 << 16);
    }();
    const uint32_t hadn = had ^ 0x80008000u;
    const float* dq = s_dq + (isq ? 0 : K);
    F2 y[M][2][2][2];  // [m][eh][row half][channel pair]: channel 32 m + 8 j + 4 eh + 2 pair + (0, 1)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      uint32_t pc[2][3][4];  // [row half][piece][channel pair of eight]
      float x[2][8];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        if (dqk || !rot) Act<T>::unpack8(raw[r][m], x[r]);
        if (dqk) {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[r][e] = __fmul_rn(x[r][e], dq[32 * m + 8 * j + e]);
          if (rot) split3(x[r], pc[r][0], pc[r][1], pc[r][2]);
        } else {
          pc[r][0][0] = raw[r][m].x; pc[r][0][1] = raw[r][m].y; pc[r][0][2] = raw[r][m].z; pc[r][0][3] = raw[r][m].w;
        }
      }
#pragma unroll
      for (int eh = 0; eh < 2; ++eh) {
        if (rot) {
          float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
          auto mma = [&](int i) {
            const uint32_t a0 = pc[0][i][2 * eh], a1 = pc[1][i][2 * eh], a2 = pc[0][i][2 * eh + 1], a3 = pc[1][i][2 * eh + 1];
            mma_bf16(d0, a0, a1, a2, a3, had, had);
            mma_bf16(d1, a0, a1, a2, a3, had, hadn);
          };
          if (dqk) {
            mma(2);
            mma(1);
            mma(0);
          } else if (F16) {
            mma_f16(d0, pc[0][0][2 * eh], pc[1][0][2 * eh], pc[0][0][2 * eh + 1], pc[1][0][2 * eh + 1], had, had);
            mma_f16(d1, pc[0][0][2 * eh], pc[1][0][2 * eh], pc[0][0][2 * eh + 1], pc[1][0][2 * eh + 1], had, hadn);
          } else {
            mma(0);
          }
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
    // The pieces of an infinity are inf and inf - inf. Every channel of a rotated row is a sum over the whole row, so any one of
    // them shows it; such rows are made again below.
    unsigned odd = 0u;  // bit 4 i: row i, bit 4 i + 1: row i + 8
    if (!KF32 && rot && dqk) {
      float y0, y1, z;
      y[0][0][0][0].get(y0, z);
      y[0][0][1][0].get(y1, z);
      odd = (__ballot_sync(0xffffffffu, !(fabsf(y0) <= 3.402823466e38f)) & 0x11111111u) |
            ((__ballot_sync(0xffffffffu, !(fabsf(y1) <= 3.402823466e38f)) & 0x11111111u) << 1);
    }
    const float inv_sq = 1.0f / a.sq[h];
    const F2 inv(inv_sq, inv_sq), scale(a.scale, a.scale);
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int t = t0 + g + 8 * r;
        uint32_t w[4];  // the eight channels, rounded to the activation dtype
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          F2& yy = y[m][p >> 1][r][p & 1];
          if constexpr (!KF32) {  // not rotated: the factor is 1 and the values are of the activation dtype
            const float2 sg = *reinterpret_cast<const float2*>(s_sgn + 32 * m + 8 * j + 2 * p);
            float x0, x1;
            mul2(yy, F2(sg.x, sg.y)).get(x0, x1);
            w[p] = Act<T>::pack2(x0, x1);
            yy = F2(Act<T>::get(w[p], 0), Act<T>::get(w[p], 1));
          }
        }
        if (isq) {
          uint32_t cd[2];
#pragma unroll
          for (int eh = 0; eh < 2; ++eh) {
            const F2 x01 = mul2(y[m][eh][r][0], scale), x23 = mul2(y[m][eh][r][1], scale);
            cd[eh] = codes4<false>(x01, x23, inv, a.qmax);
          }
          *reinterpret_cast<uint2*>(a.qq + (tile * C + t) * K + 32 * m + 8 * j) = make_uint2(cd[0], cd[1]);
        } else if constexpr (KF32) {
          float x[8];
#pragma unroll
          for (int p = 0; p < 4; ++p) y[m][p >> 1][r][p & 1].get(x[2 * p], x[2 * p + 1]);
          *reinterpret_cast<float4*>(s_k + t * LDK + 32 * m + 8 * j) = make_float4(x[0], x[1], x[2], x[3]);
          *reinterpret_cast<float4*>(s_k + t * LDK + 32 * m + 8 * j + 4) = make_float4(x[4], x[5], x[6], x[7]);
        } else {
          *reinterpret_cast<uint4*>(s_k + t * LDK + 32 * m + 8 * j) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    if constexpr (!KF32) {
      if (odd != 0u) {  // a lane per channel, the row summed in fp32
        __syncwarp();
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
          if (((odd >> (4 * (i & 7) + (i >> 3))) & 1u) == 0u) continue;
          const T* row = src + (tok0 + (size_t)(t0 + i) * a.H) * K;
          for (int n = lane; n < K; n += 32) {
            float sum = 0.f;
#pragma unroll 1
            for (int e = 0; e < K; ++e) {
              const float x = __fmul_rn(Act<T>::to(row[e]), dq[e]);
              sum += (__popc(e & n) & 1) ? -x : x;
            }
            const T v = Act<T>::from(__fmul_rn(sum, s_sgn[n]));
            if (isq) a.qq[(tile * C + t0 + i) * K + n] = (int8_t)q8(__fmul_rn(Act<T>::to(v), a.scale), inv_sq, a.qmax);
            else s_k[(t0 + i) * LDK + n] = v;
          }
        }
      }
    }
  }
  __syncthreads();

  // ---- 2. k codes: four tokens x eight channels a thread
  if (warp < 2 * M) {
    const int tg = 8 * (warp & 1) + g, n0 = 8 * (4 * (warp >> 1) + j);
    const float inv_sk = 1.0f / a.sk[h];
    const F2 inv(inv_sk, inv_sk);
    float x[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = 4 * tg + i;
      if constexpr (KF32) {
        *reinterpret_cast<float4*>(x[i]) = *reinterpret_cast<const float4*>(s_k + t * LDK + n0);
        *reinterpret_cast<float4*>(x[i] + 4) = *reinterpret_cast<const float4*>(s_k + t * LDK + n0 + 4);
      } else {
        Act<T>::unpack8(*reinterpret_cast<const uint4*>(s_k + t * LDK + n0), x[i]);
      }
      if (e_hw != 0.f) {
        const float hw = s_hw[t];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[i][e] = Act<T>::round(__fmul_rn(x[i][e], hw));
      }
      uint32_t cd[2];
#pragma unroll
      for (int eh = 0; eh < 2; ++eh) {
        const F2 x01(x[i][4 * eh], x[i][4 * eh + 1]), x23(x[i][4 * eh + 2], x[i][4 * eh + 3]);
        cd[eh] = codes4<false>(x01, x23, inv, a.qmax);
      }
      *reinterpret_cast<uint2*>(a.kl + (tile * C + kl_row_of_token(t)) * K + n0) = make_uint2(cd[0], cd[1]);
    }
    const float4 fk = *reinterpret_cast<const float4*>(s_fk + 4 * tg);
    const F2 f[4] = {F2(fk.x, fk.x), F2(fk.y, fk.y), F2(fk.z, fk.z), F2(fk.w, fk.w)};
#pragma unroll
    for (int p = 0; p < 4; ++p) {  // codes of channel pairs, then words of four tokens
      F2 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = mul2(F2(x[i][2 * p], x[i][2 * p + 1]), f[i]);
      const F2 ikw(s_ikw[n0 + 2 * p], s_ikw[n0 + 2 * p + 1]);
      const uint32_t lo = codes4<false>(w[0], w[1], ikw, a.qmax), hi = codes4<false>(w[2], w[3], ikw, a.qmax);
      *reinterpret_cast<uint32_t*>(a.kwT + (tile * K + n0 + 2 * p) * C + 4 * tg) = __byte_perm(lo, hi, 0x6420);
      *reinterpret_cast<uint32_t*>(a.kwT + (tile * K + n0 + 2 * p + 1) * C + 4 * tg) = __byte_perm(lo, hi, 0x7531);
    }
  }
  // ---- Gram matrix (strictly lower triangle): the twenty 16 x 8 tiles on and below the diagonal blocks
  for (int u = warp; u < 20; u += 8) {
    const int blk = u >> 1, I = blk < 1 ? 0 : blk < 3 ? 1 : blk < 6 ? 2 : 3, J = blk - I * (I + 1) / 2, tj = 16 * J + 8 * (u & 1);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int kk = 0; kk < K / 16; ++kk) {
      if constexpr (KF32) {  // fp32 keys: three pieces each, six products
        const float* ra = s_k + (16 * I + g) * LDK + 16 * kk + 2 * j;
        const float* rb = s_k + (tj + g) * LDK + 16 * kk + 2 * j;
        uint32_t pa[3][4], pb[3][2];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const float2 x = *reinterpret_cast<const float2*>(ra + (p & 1) * 8 * LDK + (p >> 1) * 8);
          split3_pair(F2(x.x, x.y), pa[0][p], pa[1][p], pa[2][p]);
        }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const float2 x = *reinterpret_cast<const float2*>(rb + 8 * p);
          split3_pair(F2(x.x, x.y), pb[0][p], pb[1][p], pb[2][p]);
        }
        auto mma = [&](int i, int k2) { mma_bf16(acc, pa[i][0], pa[i][1], pa[i][2], pa[i][3], pb[k2][0], pb[k2][1]); };
        mma(2, 0);
        mma(0, 2);
        mma(1, 1);
        mma(1, 0);
        mma(0, 1);
        mma(0, 0);
      } else {
        uint32_t qa[4], kb[2];
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(qa[0]), "=r"(qa[1]), "=r"(qa[2]), "=r"(qa[3])
                     : "r"(smem_u32(s_k + (16 * I + (lane & 15)) * LDK + 16 * kk + 8 * (lane >> 4))) : "memory");
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(kb[0]), "=r"(kb[1])
                     : "r"(smem_u32(s_k + (tj + (lane & 7)) * LDK + 16 * kk + 8 * ((lane >> 3) & 1))) : "memory");
        if constexpr (F16) mma_f16(acc, qa[0], qa[1], qa[2], qa[3], kb[0], kb[1]);
        else mma_bf16(acc, qa[0], qa[1], qa[2], qa[3], kb[0], kb[1]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int i = 16 * I + g + 8 * r, jj = tj + 2 * j;
      float v[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) v[e] = jj + e < i ? s_bs[i] * s_b1[jj + e] * acc[2 * r + e] * expf(s_gc[i] - s_gc[jj + e]) : 0.f;
      *reinterpret_cast<float2*>(s_G + i * 68 + jj) = make_float2(v[0], v[1]);
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // ---- 3.
  wy_solve(s_G, s_T);
  // ---- 4. W = T diag(beta^sigma exp(gc)) k  -> w_read codes;  U = T diag(beta^sigma) v  -> activation dtype
  wy_fragments2(s_T, s_cwW, s_bs, s_frag, warp, lane);  // in the place of G and T
  __syncthreads();
  {
    constexpr int NB = KF32 ? 3 : F16 ? 2 : 1;
    const int n0 = (K / 8) * warp;
    float acc[4][KS][4];
    wy_product3<KS, NB>(acc, s_frag, lane, [&](int ks, uint32_t (&bp)[NB][KS][2]) {
      if constexpr (KF32) {
#pragma unroll
        for (int nt = 0; nt < KS; ++nt)
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const float* kp = s_k + (16 * ks + 8 * s + 2 * j) * LDK + n0 + 8 * nt + g;
            split3_pair(F2(kp[0], kp[LDK]), bp[0][nt][s], bp[1][nt][s], bp[2][nt][s]);
          }
      } else {
        wy_pieces16<T, KS>(bp, s_k + 16 * ks * LDK + n0, LDK, lane);
      }
    });
    wy_store_w<T, KS>(acc, d.wq + tile * (C * K), n0, 1.0f / d.sw[h], a.qmax, lane);
  }
  wy_u<T, V>(s_frag + 30 * 32, s_v, LDV, reinterpret_cast<T*>(d.u) + tile * (size_t)(V * C), warp, lane);
}

// ------------------------------------------------------------------------------------------------ state pass
struct DeltaStateArgs {
  const int8_t *wq, *kwT;  // wq tile in MMA order: wq_offset()
  const void* u;           // [BH,NT,V,C]
  const float *fw, *gc, *skw, *sw, *sel, *sew, *ss;
  const float *gcl, *genv;  // [BH,NT,K] decay factor of the chunk (diagonal decay), [BH,NT,C] value-side write gate
  int8_t *hT, *elT;
  float* final_state;
  const float* initial_state;  // [B,H,K,V] fp32 carry entering the first chunk, or null
  int* status;
  int H, NT, V, use_g;
  float eta, qmax;
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(bar)
               : "memory");
}

// One stage of the operand ring: W tile, kwT tile, the CTA's rows of U, the per-token factors, the decay of the chunk.
template <int K, int GV>
struct DeltaStage {
  static constexpr int kW = 0, kK = 64 * K, kU = 2 * 64 * K, kF = kU + GV * 16 * 128, kG = kF + 256, kD = kG + 256, kBytes = kD + 4 * K;
};
template <int K, int KS, int GV, int NS>
constexpr size_t delta_state_smem() {
  return (size_t)NS * DeltaStage<K, GV>::kBytes + GV * 2048 + GV * KS * 8 * 512 + 16 * NS + 4 * K;
}

// A group of KS warps owns 16 value rows of the state; a warp keeps K / KS key channels of the fp32 carry in registers (rows
// g, g + 8; eight channels 32 b + 8j .. per lane and 32-channel block b). Everything is laid out so that the codes a lane
// makes are the MMA fragment it needs next:
//   * the read is computed transposed, ws^T = hq . W^T: A = the lane's own codes of the carry, B = rows of the W tile, whose
//     tokens are dealt to the MMA columns so that a lane ends up with consecutive tokens of its two value rows;
//   * a warp contracts its own channels; the KS partial sums cross through shared memory, each warp finishing the E codes of
//     TE = 16 / KS tokens per (row, lane), and the e_write codes cross back the same way: two barriers of KS warps a step;
//   * the write product's A operand is one 16-byte read of those codes per row, its B operand rows of the kwT tile, whose
//     channels are dealt to the columns so that the lane gets its own carry channels back.
// One more warp brings the tiles by bulk copies in a ring of NS stages (every tile is contiguous in the workspace), shared by
// the GV groups of the CTA. The step is serial over the chunks: bound by its latency with few (b, h), by instruction issue
// with many (about 400 instructions per warp and step; shared memory 40 %, ALU pipe 26 % busy). Measured at K = V = 128
// against one CTA per 32 value rows with E codes stored bytewise and two block barriers per step: 25.6 -> 15.5 us at 16
// (b, h) x 16 chunks, 280 -> 240 us at 64 x 128; diagonal decay 54 -> 38 us at 32 x 31, 994 -> 720 us at 256 x 128.
// Every wait is bounded; on expiry the CTA raises the status word, stores nothing more and waits no more.
template <typename T, int K, int KS, int GV, int NS, int MINB, bool DIAG, bool Q127>
__global__ void __launch_bounds__(32 * (KS * GV + 1), MINB) zoo_state_delta_kernel(DeltaStateArgs a) {
  pdl_enter();
  constexpr int C = 64, NB = K / 32 / KS, NTE = 8 / KS, TE = 2 * NTE;
  static_assert(KS == 2 || KS == 4, "a group is two or four warps");
  typedef DeltaStage<K, GV> S;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint8_t* s_stage = smem_raw;                                  // [NS][S::kBytes]
  uint8_t* s_codes = s_stage + NS * S::kBytes;                  // [GV][e_write | e_local][16][C]
  int4* s_part = reinterpret_cast<int4*>(s_codes + GV * 2048);  // [GV][from][n-tile][lane]
  const uint32_t bars = smem_u32(s_codes + GV * 2048 + GV * KS * 8 * 512);  // full[NS], empty[NS]
  float* s_skw = reinterpret_cast<float*>(s_codes + GV * 2048 + GV * KS * 8 * 512 + 16 * NS);  // [K]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh = blockIdx.y, h = bh % a.H;
  const int V = a.V, v0 = 16 * GV * blockIdx.x;
  const size_t tile0 = (size_t)bh * a.NT;
  const bool gate = a.eta != 0.f && (DIAG || a.use_g);  // genv holds a factor other than 1
  for (int i = threadIdx.x; i < K; i += 32 * (KS * GV + 1)) s_skw[i] = a.skw[h * K + i];
  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bars + 8 * i));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bars + 8 * (NS + i)), "r"(KS * GV));
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();

  if (warp == KS * GV) {
    if (lane == 0) {
      bool ok = true;
      int issued = 0;
      for (int c = 0; c < a.NT && ok; ++c) {
        const int slot = c % NS;
        if (c >= NS) ok = mbar_wait_bounded(bars + 8 * (NS + slot), (c / NS - 1) & 1);
        if (!ok) break;
        const uint32_t st = smem_u32(s_stage) + slot * S::kBytes, bar = bars + 8 * slot;
        const size_t tile = tile0 + c;
        const uint32_t bytes = 2 * C * K + GV * 16 * 128 + 256 + (gate ? 256 : 0) + (DIAG ? 4 * K : (a.use_g ? 16 : 0));
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
        bulk_load(st + S::kW, a.wq + tile * (C * K), C * K, bar);
        bulk_load(st + S::kU, reinterpret_cast<const T*>(a.u) + (tile * V + v0) * C, GV * 16 * 128, bar);
        bulk_load(st + S::kF, a.fw + tile * C, 256, bar);
        if (gate) bulk_load(st + S::kG, a.genv + tile * C, 256, bar);
        bulk_load(st + S::kK, a.kwT + tile * (K * C), K * C, bar);
        if (DIAG) bulk_load(st + S::kD, a.gcl + tile * K, 4 * K, bar);
        else if (a.use_g) bulk_load(st + S::kD, a.gc + tile * C + C - 4, 16, bar);
        ++issued;
      }
      // copies still in flight must land before the CTA may exit
      for (int c = max(0, issued - NS); c < issued; ++c) ok = mbar_wait_bounded(bars + 8 * (c % NS), (c / NS) & 1) && ok;
      if (!ok) atomicExch(a.status, 1);
    }
    return;
  }

  const int ks = warp % KS, gv = warp / KS;
  const int g = lane >> 2, j = lane & 3;
  const int va = v0 + 16 * gv + g, vb = va + 8;
  const int kc0 = 32 * NB * ks + 8 * j;  // first of the lane's eight key channels in its first block
  const int t0 = 16 * j + TE * ks;       // first of the lane's TE tokens
  auto group_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + gv), "n"(32 * KS) : "memory"); };
  F2 nsws[2], ihq[2], isel[2], isew[2], sew[2];  // per value row: -s_w s_state, 1 / s_state, 1 / s_el, 1 / s_ew, s_ew
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int v = r ? vb : va;
    const float ss = a.ss[h * V + v], n = -a.sw[h] * ss, iel = 1.0f / a.sel[h * V + v];
    const float ew = a.sew[h * V + v], iew = 1.0f / ew, ih = 1.0f / ss;
    sew[r] = F2(ew, ew);
    nsws[r] = F2(n, n); ihq[r] = F2(ih, ih); isel[r] = F2(iel, iel); isew[r] = F2(iew, iew);
  }
  F2 skw[NB == 1 ? 4 : 1], carry[NB][2][4];  // several blocks per warp: the key scales stay in shared memory
#pragma unroll
  for (int b = 0; b < NB; ++b) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = kc0 + 32 * b + 2 * i;
      if (NB == 1) skw[NB == 1 ? i : 0] = F2(s_skw[k], s_skw[k + 1]);
      const size_t r0 = ((size_t)bh * K + k) * V, r1 = r0 + V;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int v = r ? vb : va;
        carry[b][r][i] = a.initial_state ? F2(a.initial_state[r0 + v], a.initial_state[r1 + v]) : F2(0.f, 0.f);
      }
    }
  }

  bool ok = true;
  int slot = 0;
  uint32_t phase = 0;
  for (int c = 0; c < a.NT; ++c) {
    if (ok) ok = mbar_wait_bounded(bars + 8 * slot, phase);
    const uint8_t* st = s_stage + slot * S::kBytes;
    // with one channel block per warp every operand of the step is read up front: no read waits behind a barrier
    constexpr bool EARLY = NB == 1;
    const uint8_t* wrow = st + S::kW + ks * NB * 2048 + g * 32 + 8 * j;
    const uint8_t* krow = st + S::kK + (32 * NB * ks + 8 * (g >> 1) + (g & 1)) * C + 16 * j;
    uint2 wf[EARLY ? 8 : 1], uf[2][TE / 4];
    uint4 kf[EARLY ? 4 : 1];
    float4 ff[TE / 4], gf[TE / 4];
    if constexpr (EARLY) {
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) wf[nt] = *reinterpret_cast<const uint2*>(wrow + nt * 256);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) kf[nt] = *reinterpret_cast<const uint4*>(krow + 2 * nt * C);
    }
    auto read_factors = [&]() {
#pragma unroll
      for (int i4 = 0; i4 < TE / 4; ++i4) {
        ff[i4] = *reinterpret_cast<const float4*>(st + S::kF + 4 * (t0 + 4 * i4));
        if (gate) gf[i4] = *reinterpret_cast<const float4*>(st + S::kG + 4 * (t0 + 4 * i4));
#pragma unroll
        for (int r = 0; r < 2; ++r) uf[r][i4] = *reinterpret_cast<const uint2*>(st + S::kU + (16 * gv + g + 8 * r) * 128 + 2 * (t0 + 4 * i4));
      }
    };
    if (EARLY) read_factors();

    // ---- 1. INT8 copy of the carry entering the chunk: stored state and A fragments in one
    uint32_t hq[NB][2][2];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        hq[b][r][0] = codes4<true>(carry[b][r][0], carry[b][r][1], ihq[r], 127.f);
        hq[b][r][1] = codes4<true>(carry[b][r][2], carry[b][r][3], ihq[r], 127.f);
        if (ok)
          *reinterpret_cast<uint2*>(a.hT + ((tile0 + c) * V + state_row_of_channel(r ? vb : va)) * K + kc0 + 32 * b) =
              make_uint2(hq[b][r][0], hq[b][r][1]);
      }
    }

    // ---- 2. reads over this warp's channels, partial sums exchanged within the group
    int ws[NTE][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      int acc[4];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const uint2 w = EARLY ? wf[EARLY ? nt : 0] : *reinterpret_cast<const uint2*>(wrow + b * 2048 + nt * 256);
        if (b == 0) mma_s8_first(acc, hq[b][0][0], hq[b][1][0], hq[b][0][1], hq[b][1][1], w.x, w.y);
        else mma_s8(acc, hq[b][0][0], hq[b][1][0], hq[b][0][1], hq[b][1][1], w.x, w.y);
      }
      s_part[((gv * KS + ks) * 8 + nt) * 32 + lane] = make_int4(acc[0], acc[1], acc[2], acc[3]);
    }
    group_sync();
#pragma unroll
    for (int i = 0; i < NTE; ++i) {
      const int4* p = s_part + (gv * KS * 8 + NTE * ks + i) * 32 + lane;
      int4 s = p[0];
#pragma unroll
      for (int q = 1; q < KS; ++q) {
        const int4 x = p[q * 256];
        s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
      }
      ws[i][0] = s.x + 0x4B400000; ws[i][1] = s.y + 0x4B400000; ws[i][2] = s.z + 0x4B400000; ws[i][3] = s.w + 0x4B400000;
    }

    // ---- 3. E = (U - ws) fw and its codes for TE tokens of two value rows
    uint8_t* s_ew = s_codes + gv * 2048;
    if (!EARLY) read_factors();
#pragma unroll
    for (int i4 = 0; i4 < TE / 4; ++i4) {
      const F2 f01(ff[i4].x, ff[i4].y), f23(ff[i4].z, ff[i4].w);
      const F2 v01(gf[i4].x, gf[i4].y), v23(gf[i4].z, gf[i4].w);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint2 u = uf[r][i4];
        F2 E01 = fma2(unbias2(ws[2 * i4][2 * r], ws[2 * i4][2 * r + 1]), nsws[r], F2(Act<T>::get(u.x, 0), Act<T>::get(u.x, 1)));
        F2 E23 = fma2(unbias2(ws[2 * i4 + 1][2 * r], ws[2 * i4 + 1][2 * r + 1]), nsws[r], F2(Act<T>::get(u.y, 0), Act<T>::get(u.y, 1)));
        E01 = mul2(E01, f01);
        E23 = mul2(E23, f23);
        float e0, e1, e2, e3;
        E01.get(e0, e1);
        E23.get(e2, e3);
        const uint32_t p01 = Act<T>::pack2(e0, e1), p23 = Act<T>::pack2(e2, e3);  // e_local: rounded to the activation type
        uint8_t* dst = s_ew + (g + 8 * r) * C + t0 + 4 * i4;
        *reinterpret_cast<uint32_t*>(dst + 1024) = codes4<Q127>(F2(Act<T>::get(p01, 0), Act<T>::get(p01, 1)),
                                                                F2(Act<T>::get(p23, 0), Act<T>::get(p23, 1)), isel[r], a.qmax);
        if (gate) {
          E01 = mul2(E01, v01);
          E23 = mul2(E23, v23);
        }
        *reinterpret_cast<uint32_t*>(dst) = codes4<Q127>(E01, E23, isew[r], a.qmax);
      }
    }
    group_sync();

    // ---- 4. e_local rows out (1 KB per group, contiguous); write product and carry update
    {
      uint4* eout = reinterpret_cast<uint4*>(a.elT + ((tile0 + c) * V + v0 + 16 * gv) * C);
#pragma unroll
      for (int i = ks * 32 + lane; i < 64; i += 32 * KS)
        if (ok) eout[i] = *reinterpret_cast<const uint4*>(s_ew + 1024 + 16 * i);
    }
    const uint4 ea = *reinterpret_cast<const uint4*>(s_ew + g * C + 16 * j);
    const uint4 eb = *reinterpret_cast<const uint4*>(s_ew + (g + 8) * C + 16 * j);
    const float gs = !DIAG && a.use_g ? expf(*reinterpret_cast<const float*>(st + S::kD + 12)) : 1.0f;
    const F2 gs2(gs, gs);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const uint4 k4 = EARLY ? kf[EARLY ? nt : 0] : *reinterpret_cast<const uint4*>(krow + (32 * b + 2 * nt) * C);
        int acc[4];
        mma_s8_biased(acc, ea.x, eb.x, ea.y, eb.y, k4.x, k4.y);
        mma_s8(acc, ea.z, eb.z, ea.w, eb.w, k4.z, k4.w);
        F2 gm = gs2;
        if (DIAG) gm.v = *reinterpret_cast<const unsigned long long*>(st + S::kD + 4 * (kc0 + 32 * b + 2 * nt));
        F2 sk = skw[NB == 1 ? nt : 0];
        if (NB > 1) sk.v = *reinterpret_cast<const unsigned long long*>(s_skw + kc0 + 32 * b + 2 * nt);
        carry[b][0][nt] = fma2(carry[b][0][nt], gm, mul2(mul2(unbias2(acc[0], acc[1]), sk), sew[0]));
        carry[b][1][nt] = fma2(carry[b][1][nt], gm, mul2(mul2(unbias2(acc[2], acc[3]), sk), sew[1]));
      }
    }
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bars + 8 * (NS + slot)) : "memory");
    if (++slot == NS) { slot = 0; phase ^= 1; }
  }
  if (!ok) atomicExch(a.status, 1);

  if (a.final_state != nullptr && ok) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float* r0 = a.final_state + ((size_t)bh * K + kc0 + 32 * b + 2 * i) * V;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          float x, y;
          carry[b][r][i].get(x, y);
          r0[r ? vb : va] = x;
          r0[V + (r ? vb : va)] = y;
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ state pass, canonical storage
template <int ROWB>
__device__ __forceinline__ int swz_row(int row, int chunk) {
  if (ROWB == 128) return row * 128 + ((chunk ^ ((row & 1) << 2)) << 4);
  return row * 64 + (chunk << 4);
}

// Delta-rule state pass when v arrives rotated by R_V and the state is stored canonical (zoo/gated_delta_rule.py,
// zoo/kda.py with unrot=; reference.py:218-227). Per chunk:
//   ws   = fp16(dequant(W_q . S_q)) . R_V            the canonical state read, taken into the rotated value basis
//   E    = (U - ws) * fw,   e_local / e_write codes   (E stays rotated)
//   carry <- gamma carry + fp16(dequant(kw_q^T . ew_q)) . R_V^T     the write product, un-rotated
// Both basis changes mix all value channels and the read contracts over all key channels, so one CTA owns the whole
// K x V state of a (batch, head): eight warps, warp w keeping key rows 16w .. 16w+15 x all value channels of the fp32
// carry in the accumulator layout of the un-rotation MMA. The fp16 products go through shared memory; R_V and R_V^T
// both sit in shared memory with the contraction index contiguous. This path trades parallelism (B*H CTAs) for
// exactness of the reference's rounding points.
template <typename T, int K, int V, bool DIAG>
__global__ void __launch_bounds__(256) zoo_state_delta_unrot_kernel(DeltaStateArgs a, const __half* unrot_t) {
  pdl_enter();
  constexpr int C = 64, LDH = V + 8, KK = K / 64, KW = K / 16;
  constexpr int NT2 = V / 16;                 // value n-tiles per warp in the read phase (two value halves)
  constexpr int MTV = V / 16, NHALF = 8 / MTV, NTW = (K / 8) / NHALF;  // write product: value m-tile, key n-tiles per warp
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint8_t* s_h = smem_raw;                                   // [V][K]   INT8 state, B operand of the read
  uint8_t* s_ew = s_h + V * K;                               // [V][C]   e_write codes (token index contiguous)
  uint8_t* s_el = s_ew + V * C;                              // [V][C]   e_local codes
  uint8_t* s_kw = s_el + V * C;                              // [K][C]   k_write codes of the chunk
  __half* s_r = reinterpret_cast<__half*>(s_kw + K * C);     // [V][LDH] unrot   : B operand of the read rotation (rows v', v contiguous)
  __half* s_rt = s_r + V * LDH;                              // [V][LDH] unrot^T : B operand of the write un-rotation
  __half* s_x = s_rt + V * LDH;                              // [K][LDH] fp16 products: ws [64][LDH], then the write product [K][LDH]
  float* s_ss = reinterpret_cast<float*>(s_x + K * LDH);     // [V] state scale, then 1/state, 1/sel, 1/sew, sew
  float* s_iss = s_ss + V;
  float* s_isel = s_iss + V;
  float* s_isew = s_isel + V;
  float* s_sew = s_isew + V;
  float* s_skw = s_sew + V;                                  // [K]

  const int bh = blockIdx.x, h = bh % a.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, j = lane & 3;
  const int tw = warp & 3, vh = warp >> 2;
  const int ta = 16 * tw + g, tb = ta + 8;
  const int ka = 16 * warp + g, kb_ = ka + 8;   // carry rows (warps below KW)
  const bool owner = warp < KW;

  for (int i = tid; i < V * (V / 8); i += 256) {
    const int row = i / (V / 8), ch = i % (V / 8);
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(unrot_t + (size_t)row * V) + ch);
    *reinterpret_cast<uint4*>(s_rt + row * LDH + 8 * ch) = w;
    const __half* hv = reinterpret_cast<const __half*>(&w);
#pragma unroll
    for (int e = 0; e < 8; ++e) s_r[(8 * ch + e) * LDH + row] = hv[e];  // transposed copy
  }
  for (int i = tid; i < V; i += 256) {
    s_ss[i] = a.ss[h * V + i];
    s_iss[i] = 1.0f / a.ss[h * V + i];
    s_isel[i] = 1.0f / a.sel[h * V + i];
    s_isew[i] = 1.0f / a.sew[h * V + i];
    s_sew[i] = a.sew[h * V + i];
  }
  for (int i = tid; i < K; i += 256) s_skw[i] = a.skw[h * K + i];
  const float sw = a.sw[h];
  const size_t base_tile = (size_t)bh * a.NT;
  const T* up = reinterpret_cast<const T*>(a.u);

  float carry[V / 8][4];
#pragma unroll
  for (int nt = 0; nt < V / 8; ++nt) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int kr = (i >> 1) ? kb_ : ka;
      carry[nt][i] = (a.initial_state && owner) ? a.initial_state[((size_t)bh * K + kr) * V + 8 * nt + 2 * j + (i & 1)] : 0.f;
    }
  }

  auto stage_kw = [&](int c) {
    const int8_t* kwc = a.kwT + (base_tile + c) * (size_t)(K * C);
    for (int i = tid; i < K * C / 16; i += 256) cp_async16(s_kw + 16 * i, kwc + 16 * i);
    cp_async_commit();
  };
  stage_kw(0);
  __syncthreads();

  for (int c = 0; c < a.NT; ++c) {
    const size_t tile = base_tile + c;
    // operands of the read phase (token rows ta, tb)
    uint4 wa[KK], wb[KK];
    {
      const int8_t* wqc = a.wq + tile * (size_t)(C * K);
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
        wa[kk] = __ldg(reinterpret_cast<const uint4*>(wqc + wq_offset(ta, 64 * kk + 16 * j)));
        wb[kk] = __ldg(reinterpret_cast<const uint4*>(wqc + wq_offset(tb, 64 * kk + 16 * j)));
      }
    }
    const float fwa = __ldg(a.fw + tile * C + ta), fwb = __ldg(a.fw + tile * C + tb);
    float gca, gcb, glast = 0.f;
    if (DIAG) {
      gca = __ldg(a.genv + tile * C + ta);
      gcb = __ldg(a.genv + tile * C + tb);
    } else {
      gca = a.use_g ? __ldg(a.gc + tile * C + ta) : 0.f;
      gcb = a.use_g ? __ldg(a.gc + tile * C + tb) : 0.f;
      glast = a.use_g ? __ldg(a.gc + tile * C + C - 1) : 0.f;
    }

    // ---- 1. INT8 copy of the canonical carry entering the chunk
    if (owner) {
#pragma unroll
      for (int nt = 0; nt < V / 8; ++nt) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int vc = 8 * nt + 2 * j + (i & 1), kr = (i >> 1) ? kb_ : ka;
          s_h[swz_row<K>(vc, kr >> 4) + (kr & 15)] = (uint8_t)q8(carry[nt][i], s_iss[vc], 127.f);
        }
      }
    }
    __syncthreads();
    {
      int8_t* hc = a.hT + tile * (size_t)(V * K);
      for (int i = tid; i < V * (K / 16); i += 256) {
        const int vr = i / (K / 16), ch = i % (K / 16);
        *reinterpret_cast<uint4*>(hc + (size_t)state_row_of_channel(vr) * K + 16 * ch) =
            *reinterpret_cast<const uint4*>(s_h + swz_row<K>(vr, ch));
      }
    }

    // ---- 2. ws = wq . hq, dequantised, fp16, token-major
    {
#pragma unroll
      for (int n2 = 0; n2 < NT2; ++n2) {
        const int nt = NT2 * vh + n2;
        int acc[4] = {0, 0, 0, 0};
        const int vr = 8 * nt + g;
#pragma unroll
        for (int kk = 0; kk < KK; ++kk) {
          const uint4 bs = *reinterpret_cast<const uint4*>(s_h + swz_row<K>(vr, 4 * kk + j));
          mma_s8(acc, wa[kk].x, wb[kk].x, wa[kk].y, wb[kk].y, bs.x, bs.y);
          mma_s8(acc, wa[kk].z, wb[kk].z, wa[kk].w, wb[kk].w, bs.z, bs.w);
        }
        const int vc = 8 * nt + 2 * j;
        const float s0 = s_ss[vc], s1 = s_ss[vc + 1];
        *reinterpret_cast<uint32_t*>(s_x + ta * LDH + vc) =
            Act<__half>::pack2(__fmul_rn(__fmul_rn((float)acc[0], sw), s0), __fmul_rn(__fmul_rn((float)acc[1], sw), s1));
        *reinterpret_cast<uint32_t*>(s_x + tb * LDH + vc) =
            Act<__half>::pack2(__fmul_rn(__fmul_rn((float)acc[2], sw), s0), __fmul_rn(__fmul_rn((float)acc[3], sw), s1));
      }
    }
    __syncthreads();

    // ---- 3. read rotation, E, codes
    {
      const float fva = DIAG ? gca : (a.use_g ? expf(a.eta * (glast - gca)) : 1.f);
      const float fvb = DIAG ? gcb : (a.use_g ? expf(a.eta * (glast - gcb)) : 1.f);
#pragma unroll
      for (int n2 = 0; n2 < NT2; ++n2) {
        const int nt = NT2 * vh + n2;
        float u[4] = {0.f, 0.f, 0.f, 0.f};
        const __half* brow = s_r + (8 * nt + g) * LDH;
#pragma unroll
        for (int kk = 0; kk < V / 16; ++kk) {
          const uint32_t a0 = *reinterpret_cast<const uint32_t*>(s_x + ta * LDH + 16 * kk + 2 * j);
          const uint32_t a1 = *reinterpret_cast<const uint32_t*>(s_x + tb * LDH + 16 * kk + 2 * j);
          const uint32_t a2 = *reinterpret_cast<const uint32_t*>(s_x + ta * LDH + 16 * kk + 8 + 2 * j);
          const uint32_t a3 = *reinterpret_cast<const uint32_t*>(s_x + tb * LDH + 16 * kk + 8 + 2 * j);
          mma_f16(u, a0, a1, a2, a3, *reinterpret_cast<const uint32_t*>(brow + 16 * kk + 2 * j),
                  *reinterpret_cast<const uint32_t*>(brow + 16 * kk + 8 + 2 * j));
        }
        const int vc = 8 * nt + 2 * j;
        const T* uc = up + (tile * V + vc) * C;
        const float Ua[2] = {Act<T>::to(uc[ta]), Act<T>::to(uc[C + ta])}, Ub[2] = {Act<T>::to(uc[tb]), Act<T>::to(uc[C + tb])};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int vl = vc + e;
          const float Ea = __fmul_rn(__fsub_rn(Ua[e], u[e]), fwa);
          const float Eb = __fmul_rn(__fsub_rn(Ub[e], u[2 + e]), fwb);
          s_el[vl * C + ta] = (uint8_t)q8(Act<T>::round(Ea), s_isel[vl], a.qmax);
          s_el[vl * C + tb] = (uint8_t)q8(Act<T>::round(Eb), s_isel[vl], a.qmax);
          s_ew[vl * C + ta] = (uint8_t)q8(__fmul_rn(Ea, fva), s_isew[vl], a.qmax);
          s_ew[vl * C + tb] = (uint8_t)q8(__fmul_rn(Eb, fvb), s_isew[vl], a.qmax);
        }
      }
    }
    cp_async_wait<0>();  // this chunk's k_write tile
    __syncthreads();

    // ---- 4. e_local tile out; write product in the rotated basis, dequantised, fp16, key-major
    {
      uint4* eout = reinterpret_cast<uint4*>(a.elT + tile * (size_t)(V * C));
      for (int i = tid; i < V * C / 16; i += 256) eout[i] = reinterpret_cast<const uint4*>(s_el)[i];
      const int mtv = warp % MTV, nhf = warp / MTV;
      const int va = 16 * mtv + g, vb = va + 8;
      const uint4 ea = *reinterpret_cast<const uint4*>(s_ew + va * C + 16 * j);
      const uint4 eb = *reinterpret_cast<const uint4*>(s_ew + vb * C + 16 * j);
      const float sewa = s_sew[va], sewb = s_sew[vb];
#pragma unroll
      for (int n2 = 0; n2 < NTW; ++n2) {
        const int nt = NTW * nhf + n2;
        const uint4 kq = *reinterpret_cast<const uint4*>(s_kw + (8 * nt + g) * C + 16 * j);
        int acc[4] = {0, 0, 0, 0};
        mma_s8(acc, ea.x, eb.x, ea.y, eb.y, kq.x, kq.y);
        mma_s8(acc, ea.z, eb.z, ea.w, eb.w, kq.z, kq.w);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int kc = 8 * nt + 2 * j + e;
          const float sk = s_skw[kc];
          s_x[kc * LDH + va] = __float2half_rn(__fmul_rn(__fmul_rn((float)acc[e], sk), sewa));
          s_x[kc * LDH + vb] = __float2half_rn(__fmul_rn(__fmul_rn((float)acc[2 + e], sk), sewb));
        }
      }
    }
    __syncthreads();
    if (c + 1 < a.NT) stage_kw(c + 1);  // the k_write tile of the next chunk travels during the un-rotation

    // ---- 5. un-rotation of the write product, folded into the canonical carry
    if (owner) {
      float gam[2] = {1.f, 1.f};
      if (DIAG) {
        gam[0] = __ldg(a.gcl + tile * K + ka);
        gam[1] = __ldg(a.gcl + tile * K + kb_);
      } else if (a.use_g) {
        gam[0] = gam[1] = expf(glast);
      }
#pragma unroll
      for (int nt = 0; nt < V / 8; ++nt) {
        float u[4] = {0.f, 0.f, 0.f, 0.f};
        const __half* brow = s_rt + (8 * nt + g) * LDH;
#pragma unroll
        for (int kk = 0; kk < V / 16; ++kk) {
          const uint32_t a0 = *reinterpret_cast<const uint32_t*>(s_x + ka * LDH + 16 * kk + 2 * j);
          const uint32_t a1 = *reinterpret_cast<const uint32_t*>(s_x + kb_ * LDH + 16 * kk + 2 * j);
          const uint32_t a2 = *reinterpret_cast<const uint32_t*>(s_x + ka * LDH + 16 * kk + 8 + 2 * j);
          const uint32_t a3 = *reinterpret_cast<const uint32_t*>(s_x + kb_ * LDH + 16 * kk + 8 + 2 * j);
          mma_f16(u, a0, a1, a2, a3, *reinterpret_cast<const uint32_t*>(brow + 16 * kk + 2 * j),
                  *reinterpret_cast<const uint32_t*>(brow + 16 * kk + 8 + 2 * j));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) carry[nt][i] = fmaf(carry[nt][i], gam[i >> 1], u[i]);
      }
    }
    __syncthreads();
  }

  if (a.final_state != nullptr && owner) {
    float* fs = a.final_state + (size_t)bh * K * V;
#pragma unroll
    for (int nt = 0; nt < V / 8; ++nt) {
#pragma unroll
      for (int i = 0; i < 4; ++i) fs[(size_t)((i >> 1) ? kb_ : ka) * V + 8 * nt + 2 * j + (i & 1)] = carry[nt][i];
    }
  }
}

int validate_zoo_problem(const lq_zoo_problem* p, bool delta, bool diagonal);
void fill_prologue_args(const lq_zoo_problem* p, const lq_zoo_workspace* ws, PrologueArgs& a);

template <typename T, int K, int V>
static int launch_delta_prep(const DeltaPrepArgs& d, int BH, cudaStream_t st) {
  const dim3 grid(d.pro.NT, BH);
  const bool kf32 = d.pro.dqk != nullptr && d.pro.signs == nullptr;  // rescaled and not rotated: the keys are not rounded
  const cudaError_t e = kf32 ? launch_opt_in(zoo_prologue_delta_kernel<T, K, V, true>, grid, 256, DeltaPrepSmem<T, K, V, true>::kBytes, st, d)
                             : launch_opt_in(zoo_prologue_delta_kernel<T, K, V, false>, grid, 256, DeltaPrepSmem<T, K, V, false>::kBytes, st, d);
  if (e != cudaSuccess) return fail(LQ_ERR_LAUNCH, "delta prologue: launch failed: %s", cudaGetErrorString(e));
  return check_launch("zoo_prologue_delta_kernel");
}

template <typename T>
static int dispatch_delta_prep(const lq_zoo_problem* p, const DeltaPrepArgs& d, cudaStream_t st) {
  const int BH = p->B * p->H;
  if (p->K == 64 && p->V == 64) return launch_delta_prep<T, 64, 64>(d, BH, st);
  if (p->K == 64 && p->V == 128) return launch_delta_prep<T, 64, 128>(d, BH, st);
  if (p->K == 128 && p->V == 64) return launch_delta_prep<T, 128, 64>(d, BH, st);
  if (p->K == 128 && p->V == 128) return launch_delta_prep<T, 128, 128>(d, BH, st);
  return fail(LQ_ERR_UNSUPPORTED, "delta prologue: K and V must be 64 or 128");
}

int run_prologue_delta(const lq_zoo_problem* p, const lq_zoo_workspace* ws, cudaStream_t st) {
  DeltaPrepArgs d;
  fill_prologue_args(p, ws, d.pro);
  d.beta = p->beta; d.sw = p->sw; d.wq = ws->wq; d.u = ws->u; d.fw = ws->fw; d.genv = ws->genv; d.sigma = p->sigma; d.tau = p->tau;
  if (p->act_dtype == LQ_F16) return dispatch_delta_prep<__half>(p, d, st);
  if (p->act_dtype == LQ_BF16) return dispatch_delta_prep<__nv_bfloat16>(p, d, st);
  return fail(LQ_ERR_UNSUPPORTED, "delta prologue: activation dtype must be f16 or bf16");
}

template <typename T, int K, int V>
static int launch_delta_state_unrot(const lq_zoo_problem* p, const DeltaStateArgs& a, cudaStream_t st) {
  const size_t smem = (size_t)V * K + 2 * (size_t)V * 64 + (size_t)K * 64 + sizeof(__half) * (size_t)(2 * V + K) * (V + 8) +
                      sizeof(float) * (5 * V + K);
  const __half* rt = reinterpret_cast<const __half*>(p->unrot_t);
  cudaError_t e;
  if (p->decay == LQ_DECAY_DIAGONAL) {
    e = cudaFuncSetAttribute(zoo_state_delta_unrot_kernel<T, K, V, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) launch(zoo_state_delta_unrot_kernel<T, K, V, true>, p->B * p->H, 256, smem, st, a, rt);
  } else {
    e = cudaFuncSetAttribute(zoo_state_delta_unrot_kernel<T, K, V, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) launch(zoo_state_delta_unrot_kernel<T, K, V, false>, p->B * p->H, 256, smem, st, a, rt);
  }
  if (e != cudaSuccess) return fail(LQ_ERR_LAUNCH, "delta state (canonical storage): shared memory opt-in failed: %s", cudaGetErrorString(e));
  return check_launch("zoo_state_delta_unrot_kernel");
}

template <typename T, int K, bool Q127, int KS_, int GV, int NS, int MINB>
static cudaError_t launch_delta_state_v(const lq_zoo_problem* p, const DeltaStateArgs& a, cudaStream_t st) {
  constexpr int KS = KS_ < K / 32 ? KS_ : K / 32;
  const dim3 grid(p->V / 16 / GV, p->B * p->H);
  constexpr size_t smem = delta_state_smem<K, KS, GV, NS>();
  if (p->decay == LQ_DECAY_DIAGONAL) return launch_opt_in(zoo_state_delta_kernel<T, K, KS, GV, NS, MINB, true, Q127>, grid, 32 * (KS * GV + 1), smem, st, a);
  return launch_opt_in(zoo_state_delta_kernel<T, K, KS, GV, NS, MINB, false, Q127>, grid, 32 * (KS * GV + 1), smem, st, a);
}
template <typename T, int K, bool Q127>
static cudaError_t launch_delta_state(const lq_zoo_problem* p, const DeltaStateArgs& a, cudaStream_t st) {
  // Up to two groups of 16 value rows per SM: one group per CTA, a warp per 32 key channels (the shortest step). More: two
  // warps per group and two groups per CTA (fewer instructions per group; three CTAs per SM).
  if ((long long)p->B * p->H * (p->V / 16) <= 2 * sm_count()) return launch_delta_state_v<T, K, Q127, 4, 1, 2, 1>(p, a, st);
  return launch_delta_state_v<T, K, Q127, 2, 2, 2, 3>(p, a, st);
}

template <typename T>
static int dispatch_delta_state(const lq_zoo_problem* p, const DeltaStateArgs& a, cudaStream_t st) {
  if (p->unrot_t != nullptr) {  // canonical storage: one CTA per (batch, head) owns the whole state
    if (p->K == 64 && p->V == 64) return launch_delta_state_unrot<T, 64, 64>(p, a, st);
    if (p->K == 64 && p->V == 128) return launch_delta_state_unrot<T, 64, 128>(p, a, st);
    if (p->K == 128 && p->V == 64) return launch_delta_state_unrot<T, 128, 64>(p, a, st);
    if (p->K == 128 && p->V == 128) return launch_delta_state_unrot<T, 128, 128>(p, a, st);
    return fail(LQ_ERR_UNSUPPORTED, "delta state: K and V must be 64 or 128");
  }
  const bool q127 = p->qmax == 127.f;
  cudaError_t e;
  if (p->K == 64) e = q127 ? launch_delta_state<T, 64, true>(p, a, st) : launch_delta_state<T, 64, false>(p, a, st);
  else if (p->K == 128) e = q127 ? launch_delta_state<T, 128, true>(p, a, st) : launch_delta_state<T, 128, false>(p, a, st);
  else return fail(LQ_ERR_UNSUPPORTED, "delta state: K and V must be 64 or 128");
  if (e != cudaSuccess) return fail(LQ_ERR_LAUNCH, "zoo_state_delta_kernel: %s", cudaGetErrorString(e));
  return check_launch("zoo_state_delta_kernel");
}

int run_state_delta(const lq_zoo_problem* p, const lq_zoo_workspace* ws, cudaStream_t st) {
  DeltaStateArgs a;
  a.wq = ws->wq; a.kwT = ws->kwT; a.u = ws->u; a.fw = ws->fw; a.gc = ws->gc;
  a.skw = p->skw; a.sw = p->sw; a.sel = p->sel; a.sew = p->sew; a.ss = p->sstate;
  a.hT = ws->hT; a.elT = ws->vlT; a.status = p->status != nullptr ? p->status : ws->status;
  a.final_state = p->final_state; a.initial_state = p->initial_state; a.gcl = ws->gcl; a.genv = ws->genv;
  a.H = p->H; a.NT = p->T / p->chunk; a.V = p->V; a.use_g = p->g != nullptr; a.eta = p->eta; a.qmax = p->qmax;
  if (p->act_dtype == LQ_F16) return dispatch_delta_state<__half>(p, a, st);
  if (p->act_dtype == LQ_BF16) return dispatch_delta_state<__nv_bfloat16>(p, a, st);
  return fail(LQ_ERR_UNSUPPORTED, "delta state: activation dtype must be f16 or bf16");
}

}  // namespace lq

extern "C" int lq_zoo_prologue_delta(const lq_zoo_problem* p, const lq_zoo_workspace* ws, lq_stream stream) {
  if (int e = lq::validate_zoo_problem(p, true, false)) return e;
  if (!ws) return lq::fail(LQ_ERR_NULL, "delta prologue: workspace descriptor is null");
  return lq::run_prologue_delta(p, ws, (cudaStream_t)stream);
}

extern "C" int lq_zoo_state_delta(const lq_zoo_problem* p, const lq_zoo_workspace* ws, lq_stream stream) {
  if (int e = lq::validate_zoo_problem(p, true, p && p->decay == LQ_DECAY_DIAGONAL)) return e;
  if (!ws) return lq::fail(LQ_ERR_NULL, "delta state: workspace descriptor is null");
  return lq::run_state_delta(p, ws, (cudaStream_t)stream);
}
