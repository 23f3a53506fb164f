// Linear-family prologue, tensor-core version (used when no D_QK rescale is requested).
//
// Same outputs as zoo_prologue_linear_kernel, different machine mapping:
//  * a warp owns 16 tokens of q or of k. The transform is split over the channel bits: bits 0, 1, 3, 4 are the sixteen slots of
//    an m16n8k16 product with the +-1 matrix (exact operands, fp32 accumulate), the others a butterfly between a lane's own
//    registers;
//  * MMA rows are mapped to tokens (2g, 2g+1) and a lane holds eight consecutive channels of both: row-major code tiles leave
//    as 64-bit stores, transposed tiles as 16-bit stores into the shared-memory transposer;
//  * the code rule keeps its arithmetic (fp32 x*inv, clamp, +-0.5, truncate) but saturates the upper side in the
//    pack instruction, two values to an instruction where there is one, and a CTA walks several chunks so the scale staging is
//    amortised.
// Bound by instruction issue. With the whole rotation as products (eight times as many of them) and codes one at a time, 64 (b, h) x
// 64 chunks at K = V = 128 took 113 us; this form takes 102.
// Arithmetic and references as in lq_zoo_prologue.cu.
#include <type_traits>

#include "lq_zoo_rows.cuh"

namespace lq {

template <typename T>
__device__ __forceinline__ void unpack_pairs(const uint4& r, F2 (&x)[4]) {
  float f[8];
  Act<T>::unpack8(r, f);
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = F2(f[2 * i], f[2 * i + 1]);
}
// codes of channels n, n + 1 of token t (low half) and t + 1 into rows n, n + 1 of a transposer (17 words a row)
__device__ __forceinline__ void put_pair(uint32_t* row, int t, uint32_t codes) {
  const uint32_t w = __byte_perm(codes, 0u, 0x3120);
  reinterpret_cast<uint16_t*>(row)[t >> 1] = (uint16_t)w;
  reinterpret_cast<uint16_t*>(row + 17)[t >> 1] = (uint16_t)(w >> 16);
}

template <typename T, int K, int V, bool Q127>
__global__ void __launch_bounds__(256, 2) zoo_prologue_linear_mma_kernel(PrologueArgs a, int n_tiles) {
  pdl_enter();
  constexpr int C = kChunk;
  constexpr int M = K / 32, NVQ = V == 128 ? 3 : 2;
  constexpr int RAW_Q = C * K * 2, RAW_V = C * V * 2;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint32_t(*s_kw)[17] = reinterpret_cast<uint32_t(*)[17]>(smem_raw);
  uint32_t(*s_vl)[17] = s_kw + K;
  uint32_t(*s_vw)[17] = s_vl + V;
  float* s_sgn = reinterpret_cast<float*>(s_vw + V);  // [K] sign * 1/sqrt(K)
  float* s_ikw = s_sgn + K;                           // [K] 1 / skw
  float* s_ivl = s_ikw + K;                           // [V]
  float* s_ivw = s_ivl + V;                           // [V]
  // raw activation tiles (cp.async): q,k of two chunks in flight, v of one; 16-byte pieces XOR-swizzled with bit 1
  // of the token index so that the 128-bit fragment reads are conflict free
  uint8_t* s_qk = reinterpret_cast<uint8_t*>(s_ivw + V);  // [2 buf][q|k][C][K*2]
  uint8_t* s_v = s_qk + 4 * RAW_Q;                        // [C][V*2]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, j = lane & 3;
  const bool rot = a.signs != nullptr;
  const float norm = K == 64 ? 0.125f : 0.08838834764831845f;
  const T* qp = reinterpret_cast<const T*>(a.q);
  const T* kp = reinterpret_cast<const T*>(a.k);
  const T* vp = reinterpret_cast<const T*>(a.v);

  // B fragment of the +-1 matrix on the sixteen slots: (-1)^popc(s & n) for slots s = 2j, 2j + 1 and column n = g
  const uint32_t had = [&]() {
    const uint32_t one = std::is_same<T, __half>::value ? 0x3C00u : 0x3F80u;
    const uint32_t s0 = one | ((__popc((2 * j) & g) & 1) << 15), s1 = one | ((__popc((2 * j + 1) & g) & 1) << 15);
    return s0 | (s1 << 16);
  }();

  // persistent CTAs: tile t = (batch, chunk, head) with the head fastest, strided by the grid: every CTA gets the same
  // number of tiles to within one, and the CTAs in flight read all heads of the same tokens (adjacent in memory)
  // staging copies: thread -> (token row r0 + RPI it, 16-byte piece ch0); the swizzle bit of the row does not change
  // with it, so source and destination advance by constants. Tile indices are decoded once per tile (integer
  // divisions by run-time extents are the expensive part of this bookkeeping).
  constexpr int PPRK = K / 8, RPIK = 256 / PPRK, PPRV = V / 8, RPIV = 256 / PPRV;
  const int rk0 = tid / PPRK, chk0 = tid % PPRK, rv0 = tid / PPRV, chv0 = tid % PPRV;
  const uint32_t dstk0 = rk0 * (K * 2) + ((chk0 ^ (((rk0 >> 1) & 1) << 2)) << 4);
  const uint32_t dstv0 = rv0 * (V * 2) + ((chv0 ^ (((rv0 >> 1) & 1) << 2)) << 4);
  auto stage_qk = [&](int h, int c, int b, int buf) {
    uint8_t* dst = s_qk + buf * 2 * RAW_Q + dstk0;
    const size_t off = (((size_t)b * a.T + (size_t)c * C + rk0) * a.H + h) * K + 8 * chk0;
    const T* sq = qp + off;
    const T* sk = kp + off;
    const size_t step = (size_t)RPIK * a.H * K;
#pragma unroll
    for (int it = 0; it < C / RPIK; ++it) {
      cp_async16(dst + it * RPIK * (K * 2), sq);
      cp_async16(dst + RAW_Q + it * RPIK * (K * 2), sk);
      sq += step;
      sk += step;
    }
  };
  auto stage_v = [&](int h, int c, int b) {
    const T* sv = vp + (((size_t)b * a.T + (size_t)c * C + rv0) * a.H + h) * V + 8 * chv0;
    const size_t step = (size_t)RPIV * a.H * V;
#pragma unroll
    for (int it = 0; it < C / RPIV; ++it) {
      cp_async16(s_v + dstv0 + it * RPIV * (V * 2), sv);
      sv += step;
    }
  };
  auto load_g = [&](int h, int c, int b, float& g0, float& g1) {
    if (a.g == nullptr) { g0 = g1 = 0.f; return; }
    const size_t base = ((size_t)b * a.T + (size_t)c * C) * a.H + h;
    g0 = __ldg(a.g + base + (size_t)lane * a.H);
    g1 = __ldg(a.g + base + (size_t)(lane + 32) * a.H);
  };
  auto decode = [&](int t, int& h, int& c, int& b) {
    h = t % a.H;
    const int r = t / a.H;
    c = r % a.NT;
    b = r / a.NT;
  };
  const int t_begin = blockIdx.x, t_step = gridDim.x;
  if (t_begin >= n_tiles) return;
  int h, c, b, hn = 0, cn = 0, bn = 0;
  decode(t_begin, h, c, b);
  stage_qk(h, c, b, 0);
  stage_v(h, c, b);
  cp_async_commit();
  float gn0, gn1;
  load_g(h, c, b, gn0, gn1);

  const int mt = warp & 3;
  const int ta = 16 * mt + 2 * g, tb = ta + 1;  // this thread's two tokens of the m-tile
  const int swz = ((ta >> 1) & 1) << 2;         // tb shares bit 1 of the token index

  int h_staged = -1;
  float inv_sq = 1.f, inv_sk = 1.f;
  for (int t = t_begin, it = 0; t < n_tiles; t += t_step, ++it, h = hn, c = cn, b = bn) {
    const size_t tile = ((size_t)b * a.H + h) * a.NT + c;
    const int buf = it & 1;
    const bool more = t + t_step < n_tiles;
    cp_async_wait<0>();
    __syncthreads();  // raw tiles of this chunk have landed; the previous chunk's compute and copy-out are done
    if (more) {
      decode(t + t_step, hn, cn, bn);
      stage_qk(hn, cn, bn, buf ^ 1);
      cp_async_commit();
    }
    if (h != h_staged) {  // per-head channel scales (uniform branch)
      for (int i = tid; i < K; i += 256) {
        s_sgn[i] = rot ? a.signs[i] * norm : 1.0f;
        s_ikw[i] = 1.0f / a.skw[h * K + i];
      }
      for (int i = tid; i < V; i += 256) {
        s_ivl[i] = 1.0f / a.svl[h * V + i];
        s_ivw[i] = 1.0f / a.svw[h * V + i];
      }
      h_staged = h;
      inv_sq = 1.0f / a.sq[h];
      inv_sk = 1.0f / a.sk[h];
      __syncthreads();
    }
    // ---- chunk-local cumulative log-decay, per warp (double accumulate), no shared memory
    float gca, gcb, glast;
    {
      double x0 = (double)gn0, x1 = (double)gn1;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double y0 = __shfl_up_sync(0xffffffffu, x0, d), y1 = __shfl_up_sync(0xffffffffu, x1, d);
        if (lane >= d) { x0 += y0; x1 += y1; }
      }
      x1 += __shfl_sync(0xffffffffu, x0, 31);
      const float f0 = (float)x0, f1 = (float)x1;
      if (warp == 0) {
        a.gc[tile * C + lane] = f0;
        a.gc[tile * C + 32 + lane] = f1;
      }
      glast = __shfl_sync(0xffffffffu, f1, 31);
      const float sel = (mt >> 1) ? f1 : f0;
      gca = __shfl_sync(0xffffffffu, sel, ta & 31);
      gcb = __shfl_sync(0xffffffffu, sel, tb & 31);
      if (more) load_g(hn, cn, bn, gn0, gn1);
    }
    const bool use_g = a.g != nullptr;
    const float da = glast - gca, db = glast - gcb;
    // ---------------------------------------------------------------- warps 0 - 3: the rows of k; 4 - 7: of q
    {
      const bool is_q = warp >= 4;
      const uint8_t* src = s_qk + buf * 2 * RAW_Q + (is_q ? 0 : RAW_Q);
      F2 y[M][2][2][2];  // [m][eh][token a, b][channel pair]: channel 32 m + 8 j + 4 eh + 2 pair + (0, 1)
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const uint4 ra = *reinterpret_cast<const uint4*>(src + ta * (K * 2) + (((4 * m + j) ^ swz) << 4));
        const uint4 rb = *reinterpret_cast<const uint4*>(src + tb * (K * 2) + (((4 * m + j) ^ swz) << 4));
        if (rot) {
#pragma unroll
          for (int eh = 0; eh < 2; ++eh) {
            const uint32_t a0 = eh ? ra.z : ra.x, a2 = eh ? ra.w : ra.y, a1 = eh ? rb.z : rb.x, a3 = eh ? rb.w : rb.y;
            float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
            if (std::is_same<T, __half>::value) {
              mma_f16(d0, a0, a1, a2, a3, had, had);
              mma_f16(d1, a0, a1, a2, a3, had, had ^ 0x80008000u);
            } else {
              mma_bf16(d0, a0, a1, a2, a3, had, had);
              mma_bf16(d1, a0, a1, a2, a3, had, had ^ 0x80008000u);
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              y[m][eh][r][0] = F2(d0[2 * r], d0[2 * r + 1]);
              y[m][eh][r][1] = F2(d1[2 * r], d1[2 * r + 1]);
            }
          }
        } else {
          F2 xa[4], xb[4];
          unpack_pairs<T>(ra, xa);
          unpack_pairs<T>(rb, xb);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            y[m][i >> 1][0][i & 1] = xa[i];
            y[m][i >> 1][1][i & 1] = xb[i];
          }
        }
      }
      if (rot) {  // the remaining channel bits: 2 (eh), 5 and 6 (m)
        const F2 neg(-1.f, -1.f);
        auto fly = [&](F2& p, F2& q) {
          const F2 sum = add2(p, q);
          q = fma2(q, neg, p);
          p = sum;
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
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 sg = *reinterpret_cast<const float2*>(s_sgn + 32 * m + 8 * j + 2 * i);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              float x0, x1;
              mul2(y[m][i >> 1][r][i & 1], F2(sg.x, sg.y)).get(x0, x1);
              const uint32_t w = Act<T>::pack2(x0, x1);
              y[m][i >> 1][r][i & 1] = F2(Act<T>::get(w, 0), Act<T>::get(w, 1));
            }
          }
      }
      if (is_q) {
        const F2 sc(a.scale, a.scale), inv(inv_sq, inv_sq);
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            uint32_t cd[2];
#pragma unroll
            for (int eh = 0; eh < 2; ++eh) cd[eh] = codes4<Q127>(mul2(y[m][eh][r][0], sc), mul2(y[m][eh][r][1], sc), inv, a.qmax);
            *reinterpret_cast<uint2*>(a.qq + (tile * C + ta + r) * K + 32 * m + 8 * j) = make_uint2(cd[0], cd[1]);
          }
      } else {
        const float fka = use_g ? expf((1.0f - a.eta) * da) : 1.0f, fkb = use_g ? expf((1.0f - a.eta) * db) : 1.0f;
        const F2 inv(inv_sk, inv_sk), fa(fka, fka), fb(fkb, fkb);
#pragma unroll
        for (int m = 0; m < M; ++m) {
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            uint32_t cd[2];
#pragma unroll
            for (int eh = 0; eh < 2; ++eh) cd[eh] = codes4<Q127>(y[m][eh][r][0], y[m][eh][r][1], inv, a.qmax);
            *reinterpret_cast<uint2*>(a.kl + (tile * C + kl_row_of_token(ta + r)) * K + 32 * m + 8 * j) = make_uint2(cd[0], cd[1]);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int cb = 32 * m + 8 * j + 2 * i;
            const float2 ik = *reinterpret_cast<const float2*>(s_ikw + cb);
            put_pair(&s_kw[cb][0], ta, codes4<Q127>(mul2(y[m][i >> 1][0][i & 1], fa), mul2(y[m][i >> 1][1][i & 1], fb), F2(ik.x, ik.y), a.qmax));
          }
        }
      }
    }
    // ---------------------------------------------------------------- v: three quarters of the channels by the q warps, which
    // have one code tensor to make where the k warps have two
    {
      const float fva = use_g ? expf(a.eta * da) : 1.0f, fvb = use_g ? expf(a.eta * db) : 1.0f;
      const int u0 = warp >= 4 ? 0 : NVQ, u1 = warp >= 4 ? NVQ : V / 32;
#pragma unroll 1
      for (int uu = u0; uu < u1; ++uu) {
        const int cb = 32 * uu + 8 * j;
        F2 va[4], vb[4];
        unpack_pairs<T>(*reinterpret_cast<const uint4*>(s_v + ta * (V * 2) + (((cb >> 3) ^ swz) << 4)), va);
        unpack_pairs<T>(*reinterpret_cast<const uint4*>(s_v + tb * (V * 2) + (((cb >> 3) ^ swz) << 4)), vb);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 il = *reinterpret_cast<const float2*>(s_ivl + cb + 2 * i), iw = *reinterpret_cast<const float2*>(s_ivw + cb + 2 * i);
          put_pair(&s_vl[cb + 2 * i][0], ta, codes4<Q127>(va[i], vb[i], F2(il.x, il.y), a.qmax));
          put_pair(&s_vw[cb + 2 * i][0], ta, codes4<Q127>(mul2(va[i], F2(fva, fva)), mul2(vb[i], F2(fvb, fvb)), F2(iw.x, iw.y), a.qmax));
        }
      }
    }
    __syncthreads();
    if (more) {  // the single v buffer is free again
      stage_v(hn, cn, bn);
      cp_async_commit();
    }
    uint32_t* kw_out = reinterpret_cast<uint32_t*>(a.kwT + tile * (size_t)(K * C));
    for (int i = tid; i < K * 16; i += 256) kw_out[i] = s_kw[i >> 4][i & 15];
    uint32_t* vl_out = reinterpret_cast<uint32_t*>(a.vlT + tile * (size_t)(V * C));
    uint32_t* vw_out = reinterpret_cast<uint32_t*>(a.vwT + tile * (size_t)(V * C));
    for (int i = tid; i < V * 16; i += 256) {
      vl_out[i] = s_vl[i >> 4][i & 15];
      vw_out[i] = s_vw[i >> 4][i & 15];
    }
  }
}

template <typename T, int K, int V>
static int launch_mma(const lq_zoo_problem* p, const PrologueArgs& a, cudaStream_t st) {
  const int tiles = a.NT * p->B * p->H;
  // a grid that is a multiple of the head count keeps every CTA on one head (its scales are staged once)
  int ctas = 2 * sm_count();
  if (p->H <= ctas) ctas = (ctas / p->H) * p->H;
  dim3 grid(tiles < ctas ? tiles : ctas), block(256);
  const size_t smem = sizeof(uint32_t) * 17 * (K + 2 * V) + sizeof(float) * (2 * K + 2 * V) + (size_t)(4 * 64 * K * 2 + 64 * V * 2);
  cudaError_t e;
  if (p->qmax == 127.f) {
    e = cudaFuncSetAttribute(zoo_prologue_linear_mma_kernel<T, K, V, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(zoo_prologue_linear_mma_kernel<T, K, V, true>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e == cudaSuccess) launch(zoo_prologue_linear_mma_kernel<T, K, V, true>, grid, block, smem, st, a, tiles);
  } else {
    e = cudaFuncSetAttribute(zoo_prologue_linear_mma_kernel<T, K, V, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(zoo_prologue_linear_mma_kernel<T, K, V, false>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e == cudaSuccess) launch(zoo_prologue_linear_mma_kernel<T, K, V, false>, grid, block, smem, st, a, tiles);
  }
  if (e != cudaSuccess) return fail(LQ_ERR_LAUNCH, "prologue: cannot opt in to %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  return check_launch("zoo_prologue_linear_mma_kernel");
}

template <typename T>
static int dispatch_mma(const lq_zoo_problem* p, const PrologueArgs& a, cudaStream_t st) {
  if (p->K == 64 && p->V == 64) return launch_mma<T, 64, 64>(p, a, st);
  if (p->K == 64 && p->V == 128) return launch_mma<T, 64, 128>(p, a, st);
  if (p->K == 128 && p->V == 64) return launch_mma<T, 128, 64>(p, a, st);
  if (p->K == 128 && p->V == 128) return launch_mma<T, 128, 128>(p, a, st);
  return fail(LQ_ERR_UNSUPPORTED, "prologue: K and V must be 64 or 128 (got K=%d V=%d)", p->K, p->V);
}

int run_prologue_linear_mma(const lq_zoo_problem* p, const PrologueArgs& a, cudaStream_t st) {
  if (p->act_dtype == LQ_F16) return dispatch_mma<__half>(p, a, st);
  if (p->act_dtype == LQ_BF16) return dispatch_mma<__nv_bfloat16>(p, a, st);
  return fail(LQ_ERR_UNSUPPORTED, "prologue: activation dtype must be f16 or bf16");
}

}  // namespace lq
